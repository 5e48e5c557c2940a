// rmb_kernels.hpp -- host-side launchers of the search-core kernels (rmb_kernels.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include <vector>

#include "rmb_device.cuh"

namespace rmb {

// Every pair's hits in place, at the pairs' offsets.
cudaError_t launch_scan(const DevLib& L, const DevQueries& Q, int32_t ws, uint64_t pair0, uint64_t n_pairs,
                        const uint64_t* offs, SeedHit* hits, uint32_t* hit_pair, int sms, cudaStream_t st);
// Scan units: the (query, subject) pairs, or, with per_query > 0, stretches of them: first[s] .. first[s + 1]
// of a query's per_query units are subject s's, subject[u] is unit u's.
struct ScanUnits {
    const uint32_t* first = nullptr;
    const uint32_t* subject = nullptr;
    uint32_t per_query = 0;
};
// `first` for stretches that suit the launch (empty: whole pairs); step is the scan stride in bases,
// hits_per_position the expected word hits of a scan position of the longest query.
std::vector<uint32_t> scan_segments(uint32_t n_queries, const std::vector<uint32_t>& slen, uint32_t step,
                                    double hits_per_position, int sms);
// Single-pass scan: counts per unit plus the hits staged per warp (scan_stage_entries(n_units, sms)
// SeedHits of stage), then k_scan_gather puts a range of units' hits in pair order at the units' offsets.
// A set *stage_over (a warp's stretch of SCAN_STAGE_PER_WARP entries ran out) means the staged hits are
// incomplete: the caller runs launch_scan instead.  launch_pair_offsets: pairs' counts and offsets from
// their units' offsets.
constexpr uint32_t SCAN_STAGE_PER_WARP = 32768;
uint64_t scan_stage_entries(uint64_t n_units, int sms);
cudaError_t launch_scan_stage(const DevLib& L, const DevQueries& Q, int32_t ws, const ScanUnits& U, uint64_t n_units,
                              uint32_t* counts, uint32_t* stage_start, SeedHit* stage, unsigned int* stage_over, int sms,
                              cudaStream_t st, bool queue);
cudaError_t launch_scan_gather(const ScanUnits& U, uint32_t n_subjects, uint64_t unit0, uint64_t n_units,
                               const uint32_t* counts, const uint64_t* offs, const uint32_t* stage_start,
                               const SeedHit* stage, SeedHit* hits, uint32_t* hit_pair, int sms, cudaStream_t st);
cudaError_t launch_pair_offsets(const ScanUnits& U, uint32_t n_subjects, uint64_t pair0, uint64_t n_pairs,
                                const uint64_t* unit_offs, uint32_t* counts, uint64_t* offs, int sms, cudaStream_t st);
// queue: 8 bytes of device scratch (the hit queue counter; zeroed here)
cudaError_t launch_ungapped(const DevLib& L, const DevQueries& Q, const DevParams* P, int32_t ucut, uint64_t n,
                            const SeedHit* hits, const uint32_t* hit_pair, UngBox* out, int sms, cudaStream_t st,
                            unsigned long long* queue, int blocks_per_sm = 8, const uint32_t* list = nullptr,
                            const unsigned int* n_list = nullptr);
uint64_t dedup_threads(int sms);
// Bucket-parallel diagonal dedup that extends only the hits the hash admits (one warp per pair):
// flags and boxes as launch_ungapped + launch_dedup give them.
// device bytes of the fused dedup's unit lists (units_buf below) for a pair range
size_t dedup_units_bytes(uint64_t n_pairs, uint64_t n_hits, int sms);
cudaError_t launch_dedup_extend(const DevLib& L, const DevQueries& Q, const DevParams* P, int32_t ucut,
                                uint64_t pair0, uint64_t n_pairs, uint64_t n_hits, const uint64_t* offs,
                                const SeedHit* hits, UngBox* ub, uint8_t* flags, void* cells,
                                unsigned long long* queue, void* units_buf, int sms, cudaStream_t st);
size_t diag_cell_bytes();
cudaError_t launch_dedup(const DevLib& L, const DevQueries& Q, int32_t ws, int32_t ucut, uint64_t pair0,
                         uint64_t n_pairs, const uint64_t* offs, const SeedHit* hits, const UngBox* ub, uint8_t* flags,
                         uint32_t* scratch, void* cells, int sms, cudaStream_t st);
// The dedup by (pair, bucket): of launch_ungapped's boxes, or, with `leaders`, extending hits itself
// (queue and blocks_per_sm as launch_ungapped's).  buf holds bucket_dedup_bytes(n); with a null temp only temp_bytes is set.
// The range has to pass bucket_dedup_fits.
size_t bucket_dedup_bytes(uint64_t n);
bool bucket_dedup_fits(uint64_t n_pairs, uint64_t n);
cudaError_t launch_bucket_dedup(const DevLib& L, const DevQueries& Q, const DevParams* P, int32_t ws, int32_t ucut,
                                uint64_t pair0, uint64_t n_pairs, uint64_t n, const SeedHit* hits,
                                const uint32_t* hit_pair, UngBox* ub, uint8_t* flags, void* cells,
                                unsigned long long* queue, int blocks_per_sm, bool leaders, void* buf, void* temp,
                                size_t& temp_bytes, int sms, cudaStream_t st);
cudaError_t launch_prelim(const DevLib& L, const DevQueries& Q, const DevParams* P, uint64_t n, const uint32_t* list,
                          const uint32_t* idx, const SeedHit* hits, const uint32_t* hit_pair, const UngBox* ub,
                          PrelimOut* out, uint32_t* wide, unsigned int* n_wide, unsigned long long* cells, int sms,
                          cudaStream_t st);
// Whether the thread-per-extension kernel's int16 band entries and int8 score rows hold the
// parameters exactly (scores <= 127; X-drop and gap_open + gap_extend <= 8000).
// launch_prelim_stream uses n_wide[0] (overflow count) and n_wide[1] (record queue), both zeroed.
bool prelim_pack_eligible(const int32_t* matrix256, int32_t gap_open, int32_t gap_extend, int32_t xdrop_gap);
bool prelim_stream_eligible(const int32_t* matrix256, int32_t gap_open, int32_t gap_extend, int32_t xdrop_gap);
// geo: n x prelim_geo_bytes() of scratch for the per-record geometry.
size_t prelim_geo_bytes();
cudaError_t launch_prelim_prep(const DevLib& L, const DevQueries& Q, const DevParams* P, uint64_t n,
                               const uint32_t* idx, const SeedHit* hits, const uint32_t* hit_pair, const UngBox* ub,
                               void* geo, int sms, cudaStream_t st, bool pack, const unsigned int* n_dev = nullptr);
// Launch shape of the thread-per-extension DP (from rmb_tune): group of cell steps between
// row-end blocks (4, 8, 16), resident blocks per SM, widest band a thread keeps, cell budget divisor.
// Counts a graph-captured chain keeps on the device: the DP's record count (its cell budget then
// follows on the device) and, for the front-loaded order, the front's length and the order
// buffer's length (the records past the front are read from its end).
// The fused dedup's work units (built on the device from the pair offsets).
struct DedupUnits {
    unsigned long long* heavy = nullptr;  // groups of the split pairs: pair | group << 32 | log2 G << 40
    uint32_t* light = nullptr;            // pairs with hits kept whole
    unsigned int* counts = nullptr;       // [0] heavy entries, [1] light entries
    uint64_t heavy_cap = 0;
};

struct StreamDevCounts {
    const unsigned int* n = nullptr;
    const unsigned int* n_front = nullptr;
    uint64_t order_end = 0;
};
struct StreamLaunch {
    int group = 8, blocks_per_sm = 6, window = 60, budget_div = 128;
    // the packed-row kernels (prelim_pack_eligible parameters): k_prelim_pack, after k_prelim_dual where
    // `dual` is set (prelim_dual_pays), with a list of n entries and two words between them
    bool pack = false, dual = false;
    uint32_t* list = nullptr;
    unsigned int* list_ctl = nullptr;
    int gap_open = 0, gap_extend = 0, cutoff = 0;
    const uint8_t *q_dp = nullptr, *s_dp = nullptr;  // the DP copies (DevQueries, DevLib)
    uint64_t q_stride = 0, s_stride = 0;
};
// k_prelim_dual settles the records under the gapped cutoff: it pays where a word hit alone does not
// reach it.
bool prelim_dual_pays(const int32_t* matrix256, int32_t word_size, int32_t gapped_cutoff);
// The packed-row DP's copies of the sequences, dp_bytes(copies, stride) bytes: the library's two
// (bytes from plus, and reversed) and a query set's four (q and qrc, each also reversed).
uint64_t dp_bytes(int copies, uint64_t stride);
uint64_t dp_subject_stride(uint64_t bytes, uint32_t n);
cudaError_t launch_dp_subject(const uint8_t* plus, const uint64_t* off, const uint32_t* len, uint32_t n, uint8_t* out,
                              uint64_t stride, cudaStream_t st);
uint64_t dp_query_stride(uint64_t bytes, uint32_t nq);
// (*odd_host, pinned: the 32-base stretches of the queries that hold an ambiguity code other than N, counted
// in *odd, zero before and after)
cudaError_t launch_dp_query(const uint8_t* q, const uint8_t* qrc, const uint64_t* off, const uint32_t* len, uint32_t nq,
                            uint8_t* out, uint64_t stride, unsigned int* odd, unsigned int* odd_host, cudaStream_t st);
cudaError_t launch_prelim_stream(const DevParams* P, uint64_t n, const void* geo, PrelimOut* out, uint32_t* wide,
                                 unsigned int* n_wide, unsigned long long* cells, int sms, cudaStream_t st,
                                 const uint32_t* order, uint32_t* cells_out, bool plain, const StreamLaunch& cfg,
                                 StreamDevCounts dc = StreamDevCounts{});
// Learned schedule (rmb_sched.cuh).  Raw features of each record (n x SCHED_NF floats); the
// network's predicted log1p cells of every record and the records in descending predicted cost
// (order, for launch_prelim_stream; scratch: sched_order_scratch_bytes()); the network on given
// raw features.  params: SCHED_NPARAM floats on the device.
cudaError_t launch_sched_features(const DevLib& L, const DevQueries& Q, const DevParams* P, uint64_t n,
                                  const uint32_t* idx, const SeedHit* hits, const uint32_t* hit_pair, const UngBox* ub,
                                  const uint32_t* pair_hits, float* out, int sms, cudaStream_t st);
size_t sched_order_scratch_bytes();
// layout 1: the predicted-costliest ~1/32 of the records first, the rest after in reverse arrival
// order (temp: sched_front_temp_bytes(n) bytes); 2: all records in descending predicted cost
size_t sched_front_temp_bytes(uint64_t n);
// the front-loaded order's front length, on the device, in launch_sched_order's scratch
const unsigned int* sched_front_count(const void* scratch);
cudaError_t launch_sched_order(const DevLib& L, const DevQueries& Q, const DevParams* P, uint64_t n,
                               const uint32_t* idx, const SeedHit* hits, const uint32_t* hit_pair, const UngBox* ub,
                               const uint32_t* pair_hits, const float* params, float* pred, void* scratch,
                               uint32_t* order, int sms, cudaStream_t st, int layout, void* temp, size_t temp_bytes, const unsigned int* n_dev = nullptr);
cudaError_t launch_sched_predict_features(uint64_t n, const float* feats, const float* params, float* pred, int sms,
                                          cudaStream_t st);
// Records `list` (the thread kernel's overflow), one warp per extension; dres holds 2 x n_list
// int4.  Records that overflow the warp rings go to `wide` (count in n_wide[0]).
cudaError_t launch_prelim_split(const DevLib& L, const DevQueries& Q, const DevParams* P, uint32_t n_list,
                                const uint32_t* list, const uint32_t* idx, const SeedHit* hits,
                                const uint32_t* hit_pair, const UngBox* ub, int4* dres, PrelimOut* out,
                                uint32_t* wide, unsigned int* n_wide, unsigned long long* cells, int sms,
                                cudaStream_t st, const unsigned int* n_dev = nullptr);
cudaError_t launch_prelim_wide(const DevLib& L, const DevQueries& Q, const DevParams* P, uint32_t n_wide,
                               const uint32_t* wide, const uint32_t* idx, const SeedHit* hits, const uint32_t* hit_pair,
                               const UngBox* ub, PrelimOut* out, int2* band_mem, uint64_t band_cap, uint32_t threads,
                               unsigned long long* cells, unsigned int* failures, cudaStream_t st, const unsigned int* n_dev = nullptr);
// The traceback with the band in registers: `warps` (a multiple of 4) slots of traceback_pack_bytes(rows_cap)
// in scratch.  Status 4 (the window did not fit) takes launch_traceback.
bool traceback_pack_eligible(const int32_t* matrix256, int32_t gap_open, int32_t gap_extend, int32_t xdrop);
uint64_t traceback_pack_bytes(uint32_t rows_cap);
cudaError_t launch_traceback_pack(const DevLib& L, const DevQueries& Q, const DevParams* P, uint32_t n, const TbIn* in,
                                  TbOut* out, TbHalf* half, uint32_t* ops, uint32_t ops_cap, uint8_t* scratch,
                                  uint32_t rows_cap, uint32_t warps, unsigned long long* cells, bool whole,
                                  cudaStream_t st);
cudaError_t launch_traceback(const DevLib& L, const DevQueries& Q, const DevParams* P, uint32_t n, const TbIn* in,
                             TbOut* out, TbHalf* half, uint32_t* ops, uint32_t ops_cap, uint8_t* scratch,
                             uint64_t per_thread, uint64_t band_cells, uint32_t rows_cap, uint32_t threads,
                             unsigned long long* cells, bool whole, cudaStream_t st);
// The ops of the finished items of a traceback launch, packed at the host-computed offsets off[i]
// (items with status 2 are skipped), so only the ops in use cross to the host.
cudaError_t launch_gather_ops(uint32_t n, const uint32_t* ops, uint32_t ops_cap, const TbOut* out, const uint64_t* off,
                              uint32_t* dst, int sms, cudaStream_t st);

}  // namespace rmb

namespace rmb {
// Gathers, for the prelim DP results that passed the gapped cutoff, everything the host
// Phase 2a filter needs.  sel[k] indexes the prelim output array.
struct SurvivorRec {
    uint32_t pair;
    SeedHit hit;
    UngBox ub;
    PrelimOut po;
};
cudaError_t launch_gather_survivors(uint32_t n, const uint32_t* sel, const uint32_t* idx, const SeedHit* hits,
                                    const uint32_t* hit_pair, const UngBox* ub, const PrelimOut* po,
                                    SurvivorRec* out, cudaStream_t st, const unsigned int* n_dev = nullptr);
// flags[i] == want  ->  out list of i (order kept); returns the count through *n_out (device).
cudaError_t launch_select_eq(const uint8_t* flags, uint64_t n, uint8_t want, uint32_t* out, uint32_t* n_out,
                             void* temp, size_t& temp_bytes, cudaStream_t st);
// prelim score != INT32_MIN -> list of positions.
cudaError_t launch_select_prelim(const PrelimOut* po, uint64_t n, uint32_t* out, uint32_t* n_out, void* temp,
                                 size_t& temp_bytes, cudaStream_t st, const unsigned int* n_dev = nullptr);
// exclusive sum of counts[0..n) into offs[0..n] (offs[n] = total).
cudaError_t launch_offsets(const uint32_t* counts, uint64_t n, uint64_t* offs, void* temp, size_t& temp_bytes,
                           cudaStream_t st);
}  // namespace rmb

namespace rmb {
// Builds the lookup tables of nq queries on the device (Q.q/qrc/off/len/lw/cs_off/pv_off set;
// cell_start values are global offsets into cell_q, so Q.cq_off must be all zero).
// pos_off[i] = sum over earlier queries of (2 len + 1); n_pos the total; n_cells the sum of
// (4^lw + 1); n_pv the pv words.  Returns cudaErrorNotReady with temp_bytes set when temp is
// too small.  n_valid = table entries.
cudaError_t launch_lut_build(const DevQueries& Q, int32_t ws, uint32_t nq, const uint64_t* pos_off, uint64_t n_pos,
                             uint64_t n_cells, uint64_t n_pv, uint32_t* keys, uint32_t* vals, uint32_t* keys2,
                             uint32_t* vals2, uint32_t* counts, uint32_t* cs, uint32_t* cell_q, uint32_t* pv,
                             void* temp, size_t& temp_bytes, uint64_t& n_valid, cudaStream_t st);
}  // namespace rmb

namespace rmb {
cudaError_t launch_revcomp(const uint8_t* q, const uint64_t* off, const uint32_t* len, uint32_t nq, uint64_t bytes, uint8_t* rc,
                           cudaStream_t st);
// DUST masking of a query batch in segments (k_dust_segments): unit_off[i] is query i's first unit of
// `seg` starts (dust_segment_starts), rnd the first rnd_cap bases the N draw, conv, n_n, mk (zeroed),
// flags (zeroed) and ctl (two zeroed words) scratch of the queries' layout or one word a query.  qm must
// hold a copy of q and gets the masked bases; compat adds the multi-chunk path's extra masked base
// after each interval; bits (per query at word offset bits_off[i]) one bit per position inside an
// interval; either may be null.  After it ctl[0] counts the queries whose flag is set: nothing of
// them is masked, launch_dust has to take them; ctl[1] the draws the batch needs: where that is over
// rnd_cap, nothing holds and the batch runs again with more.
uint32_t dust_segment_starts(uint64_t bases, int sms);
cudaError_t launch_dust_segments(const uint8_t* q, const uint64_t* off, const uint32_t* len, uint32_t nq,
                                 const uint32_t* unit_off, uint32_t n_units, uint32_t seg, const uint8_t* rnd,
                                 uint32_t rnd_cap, uint8_t* conv, uint32_t* n_n, uint8_t* mk, uint32_t* flags,
                                 unsigned int* ctl, uint8_t* qm, bool compat, uint32_t* bits,
                                 const uint64_t* bits_off, int sms, cudaStream_t st);
// The sequential pass over the flagged queries: `scratch` holds dust_scratch_bytes(nthreads);
// overflow counts queries whose interval list overflowed.
uint32_t dust_threads(uint32_t nq, int sms);
size_t dust_scratch_bytes(uint32_t nthreads);
cudaError_t launch_dust(const uint8_t* q, const uint64_t* off, const uint32_t* len, uint32_t nq, uint8_t* qm,
                        void* scratch, uint32_t nthreads, unsigned int* overflow, bool compat, cudaStream_t st,
                        uint32_t* bits, const uint64_t* bits_off, const uint32_t* flags);
}  // namespace rmb
