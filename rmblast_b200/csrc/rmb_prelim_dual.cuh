#pragma once
// Score-only X-drop DP, two records a thread (the body of k_prelim_dual): the throughput kernel of the
// preliminary DP.  It settles the records that stay below the gapped cutoff, all but one in thousands
// on a genome against a library; a record that reaches the cutoff, outgrows the window or meets an
// ambiguity code without a score byte is listed for k_prelim_pack.
//
// The rows, coordinates and exactness are k_prelim_pack's (rmb_prelim_pack.cuh), with the two 16-bit
// halves of a register on two different records instead of two parts of a band: a thread holds the
// window of DUAL_W diagonals of two records in registers and runs a row column by column, both
// records in every packed operation, with no shuffle and no shared-memory band.  The cells of a row
// depend on each other through the gap and the running best only, one operation each, so the
// arithmetic pipe stays busy on the other ten.
//
// Bound: the half-rate integer pipe (packed add-max, byte permutes, compares; 74 % of its rate) and the
// latency of a row's chain with 12 warps an SM, what the rows in registers leave.
// A live test is one half-precision compare: the values are below 0x7c00 and not negative, so their
// order as half floats is their order as integers; the cell is then kept or cleared by a half-precision
// product with 1 or 0, and the live columns are counted into bit masks by half-precision
// multiply-adds (1024 + sums of 2^c, exact), both on the otherwise idle multiply-add pipe.  The
// threshold (running best - X) moves from column to column in its own coordinate: one add-max, and
// one multiply-add for the diagonal's gap_extend, no constant a column.
//
// Columns that are dead in all of a warp's 64 records are left out, four at a time: on the left where no
// cell of the last row lives there or in the column behind (the vertical gap's), on the right where
// no cell lives and no horizontal gap reaches in.  Of the 56 columns 16 % go so on random word hits;
// the inner ones are never dead in all 64.
//
// A record starts in a half without clearing it: its origin is set so high that what the half's last
// record left, at most its best, stays below best - X and dies at the first look; the first row's
// cells are written over it.  So the values climb from record to record, until DUAL_REBASE.
//
// Measured (B200), preliminary DP with k_prelim_pack's part: 120 queries of 60 kb 95 ms with
// k_prelim_stream (a cell step a thread, the band in shared memory), 55 with this kernel in batches
// of 4 rows, cleared at every start, 8 warps an SM and a constant a column, 44 as it is; 1,000
// contigs 414, 243 and 191 ms; 1,060 G cells/s at 0.63 warp instructions a cell (k_prelim_stream: 380 G
// at 2.4).  A window of 56 diagonals lets 0.6 % of random word hits outgrow it (48: 5 %).
//
// Rows run in batches of DUAL_ROWS (bulk of 1,000 contigs: 4 rows 227 ms, 6 213, 8 208, before the
// last of the above); records end, start and move their windows between batches.  A record that
// ends inside a batch runs on for the rest of it: past the subject's end the rows score as blocked,
// past the query's the columns do, so no best changes, and its cells are not counted.
#include "rmb_prelim_pack.cuh"

namespace rmb {

constexpr int DUAL_W = 56, DUAL_K = 26, DUAL_ROWS = 8, DUAL_SHIFT = 4, DUAL_BLOCK = 128;
// Between two looks best + origin grows past DUAL_REBASE by a window move, a record's start (PACK_STEP_MAX + 1
// and its X) and a batch's rows, 1,524 at most; a cell's diagonal lies up to 63 * 55 above: together below
// 0x7c00, where half floats stop ordering as integers.  What is left after the origin's move keeps the
// threshold above what a dead cell can reach in a row.
constexpr int32_t DUAL_REBASE = 24576, DUAL_REBASE_BY = 24064;
static_assert(DUAL_REBASE + DUAL_SHIFT * PACK_GE_MAX + PACK_STEP_MAX + 1 + PACK_XMAX + DUAL_ROWS * PACK_STEP_MAX +
                      (DUAL_W - 1) * PACK_GE_MAX < 0x7c00, "the values stay finite half floats");
static_assert(DUAL_REBASE - DUAL_REBASE_BY - PACK_XMAX > PACK_STEP_MAX, "a dead cell stays dead after the origin's move");
static_assert(DUAL_SHIFT <= 2 * DUAL_ROWS, "moves to the left lower the origin by less than the rows raise it");
constexpr int DUAL_BITS = 10;  // columns of a half-precision bit mask
constexpr int DUAL_MASKS = (DUAL_W + DUAL_BITS - 1) / DUAL_BITS;

struct DualConst {
    uint64_t q_stride, s_stride;  // as PackConst's; the same in nibbles
    const uint8_t *q_dp, *s_dp;   // the byte copies that the records point into
    const uint32_t *q_nib, *s_nib;  // their codes, eight to a word
    uint32_t neg_go;
    uint32_t one;  // 1: a factor the compiler does not see keeps an add on the multiply-add pipe
};

__device__ __forceinline__ uint32_t half_ge(uint32_t a, uint32_t b) {  // 1.0 or 0.0 per half
    uint32_t d;
    asm("set.ge.f16x2.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t half_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t half_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// eight codes from code `i` of a nibble array
__device__ __forceinline__ uint32_t nibbles_at(const uint32_t* __restrict__ base, uint64_t i) {
    const uint32_t* w = base + (i >> 3);
    return __funnelshift_r(w[0], w[1], 4u * (uint32_t)(i & 7u));
}
// nonzero where a code is 6 (another ambiguity code)
__device__ __forceinline__ uint32_t nibbles_odd(uint32_t w) { return w & (w << 1) & 0x44444444u; }

// What a record's half needs between batches only
struct DualCold {
    uint64_t b_next, a_next;  // codes of the column past the window, of the next row
    uint32_t t;
    int32_t l_score;
};

template <bool QUEUE>
__global__ void __launch_bounds__(DUAL_BLOCK, 3)
k_prelim_dual(const DevParams* __restrict__ P, const __grid_constant__ DualConst K, uint64_t n_rec,
              const PrelimGeo* __restrict__ geo, PrelimOut* __restrict__ out, uint32_t* __restrict__ list,
              unsigned int* __restrict__ n_list, unsigned int* __restrict__ queue,
              unsigned long long* __restrict__ cells_total, const uint32_t* __restrict__ order,
              uint32_t* __restrict__ cells_out, uint32_t window, StreamDevCounts dc) {
    constexpr int W = DUAL_W;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ uint2 tab[16];
    __shared__ DualCold cold[2][DUAL_BLOCK];
    const int32_t ge = P->gap_extend, go = P->gap_open, goe = go + ge, cutoff = P->gapped_cutoff;
    if (threadIdx.x < 16) {
        uint32_t b[8];
        for (int c = 0; c < 8; ++c) {
            int32_t v = threadIdx.x > 3 ? -1000 : c < 4 ? P->matrix[threadIdx.x * 16 + c] : c == 4 ? P->matrix[threadIdx.x * 16 + 14] : -1000;
            v += 2 * ge;
            b[c] = (uint32_t)(v < -128 ? -128 : v) & 0xffu;
        }
        tab[threadIdx.x] = make_uint2(b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24, b[4] | b[5] << 8 | b[6] << 16 | b[7] << 24);
    }
    __syncthreads();
    uint64_t order_end = 0;
    uint32_t n_front = 0xffffffffu;
    if (dc.n) n_rec = *dc.n;
    if (dc.n_front) {
        n_front = *dc.n_front;
        order_end = dc.order_end;
    }
    const StreamDiv div_ge(ge);
    const uint32_t step2 = pack2(2 * ge, 2 * ge), ge2 = pack2(ge, ge);

    uint32_t H[W], E[W], s[2][7];
#pragma unroll
    for (int c = 0; c < W; ++c) H[c] = E[c] = 0;
    int phase[2] = {0, 0};  // 0 needs a record, 1 left extension, 2 right extension, 4 no records left
    uint32_t pb = pack2(DUAL_REBASE - DUAL_REBASE_BY, DUAL_REBASE - DUAL_REBASE_BY), xp = 0, nx = 0;  // nx: -X  // best + origin; X
    int32_t org[2] = {0, 0}, rows[2] = {0, 0}, kr[2] = {0, 0};    // rows: rows left; kr as k_prelim_pack's
    uint32_t rec[2] = {0, 0};
    uint32_t ended = 3, failed = 0;  // bit h: half h's extension is over; it goes to the list
    unsigned long long cells = 0;
    uint32_t taken = 0;
    auto take = [&]() -> uint32_t {
        if (QUEUE) return atomicAdd(queue, 1u);
        return taken < 2 ? (blockIdx.x * DUAL_BLOCK + threadIdx.x) * 2 + taken++ : 0xffffffffu;
    };
    uint32_t next_t = take(), next_id = 0;
    bool known = false;  // next_id is next_t's record
    auto resolve = [&]() -> uint32_t {
        return !order ? next_t : next_t < n_front ? order[next_t] : order[order_end - 1 - (uint64_t)(next_t - n_front)];
    };
    uint32_t fetched = 0xffffffffu;
    uint32_t un = 0;  // live outer columns of the warp's last row: bit c of the first 13, bit c - 24 of those from 40 on
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 7; ++i) s[h][i] = 0x55555555u;

    for (;;) {
        if (__any_sync(FULL, (ended & 1u && phase[0] != 4) || (ended & 2u && phase[1] != 4))) {
            uint32_t vj = 0;  // the new halves' J
            int32_t base[2] = {0, 0};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                DualCold& k = cold[h][threadIdx.x];
                // a first step adds PACK_STEP_MAX at most to what the half still holds, all of it at most its best
                const int32_t top = (int32_t)(h ? pb >> 16 : pb & 0xffffu) + PACK_STEP_MAX + 1;
                while ((ended >> h & 1u) && phase[h] != 4) {
                    const int32_t best = (int32_t)((h ? pb >> 16 : pb & 0xffffu)) - org[h];
                    if (phase[h] != 0) {
                        if (failed >> h & 1u) {
                            list[atomicAdd(n_list, 1u)] = k.t;
                            phase[h] = 0;
                        } else if (phase[h] == 1) {
                            k.l_score = best;
                            phase[h] = 2;
                        } else {
                            const int32_t total = k.l_score + best;
                            if (total >= cutoff) {
                                list[atomicAdd(n_list, 1u)] = k.t;
                            } else {
                                out[k.t] = PrelimOut{INT32_MIN, 0, 0, 0, 0, 0, 0};
                                if (cells_out) cells_out[k.t] = rec[h];
                                cells += rec[h];
                            }
                            phase[h] = 0;
                        }
                    }
                    failed &= ~(1u << h);
                    if (phase[h] == 0) {
                        if (next_t >= n_rec) {
                            phase[h] = 4;
                            pb = h ? (pb & 0xffffu) | (uint32_t)top << 16 : (pb & 0xffff0000u) | (uint32_t)top;
                            xp &= h ? 0x0000ffffu : 0xffff0000u;
                            nx &= h ? 0x0000ffffu : 0xffff0000u;
                            break;
                        }
                        k.t = known ? next_id : resolve();
                        next_t = take();
                        known = false;
                        rec[h] = 0;
                        k.l_score = 0;
                        phase[h] = 1;
                    }
                    const uint4* gp = reinterpret_cast<const uint4*>(geo + k.t);
                    const uint4 g0 = gp[0], g1 = gp[1];
                    const int32_t X = (int32_t)reinterpret_cast<const uint32_t*>(gp)[10];
                    uint64_t ai = (((uint64_t)g0.w << 32) | g0.z) - (uint64_t)K.s_dp;
                    uint64_t bi = (((uint64_t)g0.y << 32) | g0.x) - (uint64_t)K.q_dp;
                    int32_t m = (int32_t)g1.w, nb = (int32_t)g1.z;
                    if (phase[h] == 1) {
                        ai += K.s_stride + (g1.y - g1.w);
                        bi += K.q_stride + (g1.x - g1.z);
                    } else {
                        ai += g1.w;
                        bi += g1.z;
                        m = (int32_t)g1.y - m;
                        nb = (int32_t)g1.x - nb;
                    }
                    org[h] = top + X;
                    pb = h ? (pb & 0xffffu) | (uint32_t)org[h] << 16 : (pb & 0xffff0000u) | (uint32_t)org[h];
                    if (m <= 0 || nb <= 0) continue;  // an empty extension: score 0
                    const int32_t jmax = (int32_t)div_ge((uint32_t)(X - goe)) + 1;
                    const int32_t J = jmax < nb ? jmax : nb;
                    bi -= DUAL_K;
                    const uint32_t* w = K.q_nib + (bi >> 3);
                    const uint32_t sh = 4u * (uint32_t)(bi & 7u);
                    uint32_t odd = 0, w0 = w[0];
#pragma unroll
                    for (int i = 0; i < 7; ++i) {
                        const uint32_t w1 = w[i + 1];
                        s[h][i] = __funnelshift_r(w0, w1, sh);
                        odd |= nibbles_odd(s[h][i]);
                        w0 = w1;
                    }
                    if (odd || (uint32_t)J + 1 > window) {
                        failed |= 1u << h;
                        continue;
                    }
                    k.a_next = ai;
                    k.b_next = bi + W;
                    rows[h] = m;
                    kr[h] = -DUAL_K - nb;
                    rec[h] += (uint32_t)J + 1;
                    base[h] = org[h] + ge * DUAL_K;
                    xp = h ? (xp & 0xffffu) | (uint32_t)X << 16 : (xp & 0xffff0000u) | (uint32_t)X;
                    nx = h ? (nx & 0xffffu) | (uint32_t)(-X) << 16 : (nx & 0xffff0000u) | ((uint32_t)(-X) & 0xffffu);
                    vj |= (uint32_t)J << (16 * h);
                    ended &= ~(1u << h);
                }
            }
            __syncwarp();
            if (!__any_sync(FULL, phase[0] != 4 || phase[1] != 4)) break;
            // the initial rows (gapped.rs:165-200): cell 0, gap cells 1 .. J; cell J's diagonal leads out
            // of the first row's band
            const uint32_t fresh = prmt((vj + 0x7fff7fffu), 0, 0xbb99);  // halves with a new J (J >= 1)
            const uint32_t v1 = pack2(base[0] - go, base[1] - go), v2 = pack2(base[0] - 2 * go, base[1] - 2 * go);
            H[DUAL_K] = (H[DUAL_K] & ~fresh) | (pack2(base[0], base[1]) & fresh);
            E[DUAL_K] = (E[DUAL_K] & ~fresh) | (v1 & fresh);
            uint32_t in = fresh;  // halves with gap cell i
#pragma unroll
            for (int i = 1; i <= 16; ++i) {
                const uint32_t in1 = prmt(vj + 0x80008000u - (uint32_t)(i + 1) * 0x00010001u, 0, 0xbb99);
                E[DUAL_K + i] = (E[DUAL_K + i] & ~in) | (v2 & in);
                H[DUAL_K + i] = (H[DUAL_K + i] & ~in1) | (v1 & in1);
                in = in1;
            }
            un |= 0x7u << 16;  // cells 14 .. 16 of the initial rows
        }

        // ---- the residues of a batch of rows
        uint32_t pend[2], aw[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            DualCold& k = cold[h][threadIdx.x];
            pend[h] = 0x55555555u;
            aw[h] = 0xffffffffu;
            if (phase[h] != 4) {
                pend[h] = nibbles_at(K.q_nib, k.b_next);
                aw[h] = nibbles_at(K.s_nib, k.a_next);
                k.b_next += DUAL_ROWS;
                k.a_next += DUAL_ROWS;
                if (nibbles_odd(pend[h])) {
                    ended |= 1u << h;
                    failed |= 1u << h;
                }
            }
        }
        int32_t fc[2] = {0, 0}, lc[2] = {0, 0};
#pragma unroll 1
        for (int u = 0; u < DUAL_ROWS; ++u) {
            pb += step2;
            const uint2 ta = tab[aw[0] & 15u], tb = tab[aw[1] & 15u];
            aw[0] >>= 4;
            aw[1] >>= 4;
            uint32_t w = pb - xp, f = 0, al[DUAL_MASKS];  // w: the running best - X, at the next column's diagonal
            int end = W;
#pragma unroll
            for (int i = 0; i < DUAL_MASKS; ++i) al[i] = 0x64006400u;
#pragma unroll
            for (int g = 0; g < W / 4; ++g) {
                if (g < 3 && !(un & ((1u << (4 * g + 5)) - 1u))) {
                    w += 4 * ge2;
                    continue;
                }
                if (g >= 10 && !(un >> (4 * g - 24)) && !__any_sync(FULL, half_ge(f, w) != 0)) {
                    end = 4 * g;
                    break;
                }
                const uint32_t ga = prmt(ta.x, ta.y, g & 1 ? s[0][g / 2] >> 16 : s[0][g / 2]);
                const uint32_t gb = prmt(tb.x, tb.y, g & 1 ? s[1][g / 2] >> 16 : s[1][g / 2]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = 4 * g + j;
                    const uint32_t sc = prmt(ga, gb, (uint32_t)(j | (8 | j) << 4 | (4 + j) << 8 | (12 + j) << 12));
                    const uint32_t up = c + 1 < W ? E[c + 1 < W ? c + 1 : c] : 0u;
                    const uint32_t t = __viaddmax_s16x2(H[c], sc, up);
                    const uint32_t cell = __vmaxs2(t, f);
                    f = __viaddmax_s16x2(t, K.neg_go, f);
                    const uint32_t thr = __viaddmax_s16x2(t, nx, w);
                    w = thr * K.one + ge2;
                    const uint32_t live = half_ge(cell, thr);
                    H[c] = half_mul(cell, live);
                    al[c / DUAL_BITS] = half_fma(live, (uint32_t)(0x3c00 + 0x400 * (c % DUAL_BITS)) * 0x00010001u, al[c / DUAL_BITS]);
                    E[c] = __viaddmax_s16x2(H[c], K.neg_go, up);
                }
            }
            pb = w + xp - ge2 * (uint32_t)end;
            un = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int i = 0; i < 7; ++i) s[h][i] = __funnelshift_r(s[h][i], i < 6 ? s[h][i < 6 ? i + 1 : i] : pend[h], 4);
                pend[h] >>= 4;
                // first and last live diagonal
                uint32_t m[DUAL_MASKS];
#pragma unroll
                for (int i = 0; i < DUAL_MASKS; ++i) m[i] = (h ? al[i] >> 16 : al[i]) & 0x3ffu;
                const uint32_t lo = m[0] | m[1] << 10 | m[2] << 20, hi = m[3] | m[4] << 10 | m[5] << 20;
                un |= (lo & 0x1fffu) | hi >> 10 << 16;
                fc[h] = lo ? __ffs((int)lo) - 1 : 29 + __ffs((int)hi);
                lc[h] = hi ? 61 - __clz((int)hi) : 31 - __clz((int)lo);
                --rows[h];
                ++kr[h];
                const int32_t fj = fc[h] + kr[h], width = min(lc[h] + kr[h] + 2, 1) - fj;
                if (!(ended >> h & 1u)) {
                    if ((lo | hi) == 0) {
                        ended |= 1u << h;
                    } else if (fc[h] == 0 || lc[h] == W - 1) {
                        ended |= 1u << h;
                        failed |= 1u << h;
                    } else if (fj > 0 || rows[h] <= 0) {
                        ended |= 1u << h;
                    } else {
                        rec[h] += (uint32_t)width;
                        if ((uint32_t)width > window) {
                            ended |= 1u << h;
                            failed |= 1u << h;
                        }
                    }
                }
            }
            un = __reduce_or_sync(FULL, un);
        }

        // the next record, found while rows run: its number, then its geometry's line
        if (known) {
            if (next_id != fetched && next_t < n_rec) asm volatile("prefetch.global.L1 [%0];" ::"l"(geo + next_id));
            fetched = next_id;
        } else if (next_t < n_rec) {
            next_id = resolve();
            known = true;
        }

        // ---- between the batches: records that reached the cutoff, window moves, origins
        uint32_t right = 0, left = 0, down = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            org[h] += 2 * ge * DUAL_ROWS;
            const int32_t bo = (int32_t)(h ? pb >> 16 : pb & 0xffffu);
            if (bo > DUAL_REBASE) down |= 1u << h;
            if (!(ended >> h & 1u)) {
                if (bo - org[h] + (phase[h] == 2 ? cold[h][threadIdx.x].l_score : 0) >= cutoff) {
                    ended |= 1u << h;
                    failed |= 1u << h;
                } else if (lc[h] > W - 12 && fc[h] > DUAL_SHIFT + 8) {
                    right |= 1u << h;
                } else if (fc[h] < 9 && lc[h] < W - DUAL_SHIFT - 10) {
                    left |= 1u << h;
                }
            }
        }
        if (__any_sync(FULL, right | left | down)) {
            if (__any_sync(FULL, right)) {
                un |= (un & 0x1fffu) >> DUAL_SHIFT | 0x1fffu >> (13 - DUAL_SHIFT) << (13 - DUAL_SHIFT);
                const uint32_t sel = (right & 1u ? 0x54u : 0x10u) | (right & 2u ? 0x7600u : 0x3200u);
#pragma unroll
                for (int c = 0; c < W; ++c) {
                    H[c] = prmt(H[c], c + DUAL_SHIFT < W ? H[c + DUAL_SHIFT < W ? c + DUAL_SHIFT : c] : 0u, sel);
                    E[c] = prmt(E[c], c + DUAL_SHIFT < W ? E[c + DUAL_SHIFT < W ? c + DUAL_SHIFT : c] : 0u, sel);
                }
            }
            if (__any_sync(FULL, left)) {
                un |= ((un >> 16 << DUAL_SHIFT) | ((1u << DUAL_SHIFT) - 1u)) << 16;
                const uint32_t sel = (left & 1u ? 0x54u : 0x10u) | (left & 2u ? 0x7600u : 0x3200u);
#pragma unroll
                for (int c = W - 1; c >= 0; --c) {
                    H[c] = prmt(H[c], c >= DUAL_SHIFT ? H[c >= DUAL_SHIFT ? c - DUAL_SHIFT : c] : 0u, sel);
                    E[c] = prmt(E[c], c >= DUAL_SHIFT ? E[c >= DUAL_SHIFT ? c - DUAL_SHIFT : c] : 0u, sel);
                }
            }
            uint32_t by = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                DualCold& k = cold[h][threadIdx.x];
                const int32_t move = ge * DUAL_SHIFT;
                if (right >> h & 1u) {
                    const uint32_t nw = nibbles_at(K.q_nib, k.b_next);
                    k.b_next += DUAL_SHIFT;
#pragma unroll
                    for (int i = 0; i < 7; ++i) s[h][i] = __funnelshift_r(s[h][i], i < 6 ? s[h][i < 6 ? i + 1 : i] : nw, 16);
                    kr[h] += DUAL_SHIFT;
                    org[h] += move;
                    pb += (uint32_t)move << (16 * h);
                    if (nibbles_odd(nw)) {
                        ended |= 1u << h;
                        failed |= 1u << h;
                    }
                } else if (left >> h & 1u) {
                    k.b_next -= DUAL_SHIFT;
                    const uint32_t nw = nibbles_at(K.q_nib, k.b_next - W);
#pragma unroll
                    for (int i = 6; i >= 0; --i) s[h][i] = s[h][i] << 16 | (i > 0 ? s[h][i > 0 ? i - 1 : i] >> 16 : nw & 0xffffu);
                    kr[h] -= DUAL_SHIFT;
                    org[h] -= move;
                    pb -= (uint32_t)move << (16 * h);
                    if (nibbles_odd(nw & 0xffffu)) {
                        ended |= 1u << h;
                        failed |= 1u << h;
                    }
                }
                if (down >> h & 1u) {
                    by |= (uint32_t)(0x10000 - DUAL_REBASE_BY) << (16 * h);
                    org[h] -= DUAL_REBASE_BY;
                    pb -= (uint32_t)DUAL_REBASE_BY << (16 * h);
                }
            }
            if (__any_sync(FULL, down)) {
#pragma unroll
                for (int c = 0; c < W; ++c) {
                    H[c] = __viaddmax_s16x2_relu(H[c], by, 0u);
                    E[c] = __viaddmax_s16x2_relu(E[c], by, 0u);
                }
            }
        }
    }
    if (cells) atomicAdd(cells_total, cells);
}

}  // namespace rmb
