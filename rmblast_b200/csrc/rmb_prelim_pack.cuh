#pragma once
// Score-only X-drop DP with a row's band in registers (the body of k_prelim_pack).
//
// G lanes run one extension, a row of the band a step: the band sits in a window of W = 2 G R
// diagonals (column minus row), lane l holding the diagonals 2 l R .. 2 l R + 2 R - 1 as R registers
// of two signed 16-bit values, register r the pair (2 l R + r, 2 l R + R + r).  A row is then R steps
// of packed arithmetic over all lanes, and two prefix maxima over the 2 G half-lanes: the horizontal
// gap entering a half and the running best before it.  A diagonal keeps its register from row to row,
// so the diagonal move costs nothing, the vertical gap comes from the next register, and only a path
// that drifts by gaps moves the window (by R diagonals, a register-half move).
//
// Exactness.  The reference's row (search/gapped.rs:222-296) prunes a cell below the running best,
// in row-major order, minus X, and lets the horizontal gap decay only at cells it keeps.  As in the
// warp kernels, the plain recurrence of the gap at every cell gives the same live cells, and a cell
// outside the reference's band stays dead here: left of the first live column nothing live reaches
// it, and right of the band's end only the horizontal gap does, which is the reference's extension
// of the band (gapped.rs:307-319).  In the first row the reference's band ends at the initial row's
// last cell, so that cell's diagonal is cleared.  Columns past the sequence's end score as blocked;
// gaps running past the end stay below the best and reach no column of the band.  A row whose first
// or last window diagonal is live may have lost a cell: the record goes to the warp kernel.
//
// Coordinates.  A value is held as score + gap_extend * (2 row + window diagonal) + origin, so that
// the decay of both gaps costs nothing, one packed add-max a gap; dead cells are 0 (a live value
// stays above 255) and die under every addition of a score.  The origin moves down when best + origin
// passes PACK_REBASE.
#include <cstdint>

#include "rmb_device.cuh"
#include "rmb_prelim_stream.cuh"

namespace rmb {

constexpr int PACK_BLOCK = 128;
constexpr int PACK_XMAX = 128;        // a blocked column's score is -128: it has to end any path
constexpr int PACK_STEP_MAX = 127;    // a score with both gaps' decay, 2 gap_extend, in a signed byte
constexpr int PACK_GE_MAX = 63;       // the largest gap_extend that leaves a positive score under it
constexpr int32_t PACK_REBASE = 16384, PACK_REBASE_BY = 8192;

// The launch's constants: packed pairs (the same value in both halves), by register
template <int R>
struct PackConst {
    uint64_t q_stride, s_stride;  // from the DP's copies of the sequences to the reversed ones
    uint32_t neg_go;        // -gap_open
    uint32_t neg_ge[R];     // -gap_extend * r
    uint32_t live[R];       // 0x80008000 - gap_extend * r: bit 15 of cell + live - threshold = alive
};

__host__ __device__ constexpr uint32_t pack2(int32_t lo, int32_t hi) {
    return ((uint32_t)lo & 0xffffu) | ((uint32_t)hi << 16);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
    return d;
}

// The DP's own copies of the sequences (k_dp_subject, k_dp_query): a subject base is its byte offset in
// the kernel's score table; a query base is the selector byte of its column: its score byte in a row
// of that table (code 0-3 the bases, 4 N, 5 blocked, 6 another ambiguity code) and that byte's sign,
// as prmt nibbles.  Each is also kept in reverse, so that an extension to the left reads upwards too,
// and PACK_PAD blocked columns stand at both ends of a query (a window reads past them unchecked),
// PACK_SPAD bases of code 15 between the subjects.
constexpr uint32_t PACK_PAD = 128, PACK_SPAD = 16;  // bases around each query, each subject
constexpr uint32_t PACK_BLOCKED = 5 * 17 + 128;
__host__ __device__ __forceinline__ uint32_t pack_sel(uint32_t base) {
    return (base < 4 ? base : base == 14 ? 4u : 6u) * 17u + 128u;
}
// nonzero where a byte is code 6: bits 5 and 6 set, as in no other selector byte
__device__ __forceinline__ uint32_t pack_odd(uint32_t w) { return w & (w << 1) & 0x40404040u; }

// An extension's result in three words of its record's PrelimOut (left 0-2, right 3-5) until
// k_prelim_pack_join: score; rows and columns to the best (21 bits each, the record's cells are at
// most STREAM_MAX_CELLS = 2^20 and a window) and cells (22 bits).  Half-word 12 + side is the status.
struct PackSide {
    int32_t score;
    uint32_t a, b, cells;
};
__device__ __forceinline__ void pack_store(PrelimOut* out, int side, const PackSide& r, bool ok) {
    uint32_t* w = reinterpret_cast<uint32_t*>(out) + 3 * side;
    w[0] = (uint32_t)r.score;
    w[1] = r.a | r.b << 21;
    w[2] = r.b >> 11 | r.cells << 10;
    reinterpret_cast<uint16_t*>(out)[12 + side] = ok ? 1 : 0;
}
__device__ __forceinline__ PackSide pack_side(const PrelimOut* out, int side) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(out) + 3 * side;
    return PackSide{(int32_t)w[0], w[1] & 0x1fffffu, w[1] >> 21 | (w[2] & 0x3ffu) << 11, w[2] >> 10};
}

// One extension per group of G lanes, groups fed from a queue: item 2 i is record i's left extension,
// item 2 i + 1 its right one, of the n_rec records or, with `list`, of the *n_list listed ones.  The
// records that get here after k_prelim_dual are few and long (a row waits for the one before, so the
// launch lasts as long as its longest extension): the two extensions of a record run side by side, and
// the column of the best is looked for once, in a copy of the best's row.  The records that
// k_prelim_warp_dir took here before (60 kb against 2,000 consensi) held it for 2.9 ms, 1.8 now.
template <int G, int R>
__global__ void __launch_bounds__(PACK_BLOCK)
k_prelim_pack(const DevParams* __restrict__ P, const __grid_constant__ PackConst<R> K, uint64_t n_rec,
              const PrelimGeo* __restrict__ geo, PrelimOut* __restrict__ out, unsigned int* __restrict__ queue,
              uint32_t max_cells, uint32_t window, const unsigned int* __restrict__ n_dev,
              const uint32_t* __restrict__ list, const unsigned int* __restrict__ n_list) {
    constexpr int W = 2 * G * R;
    constexpr int K_OFF = W / 2 - 2;  // the window diagonal of the pivot's diagonal at the start
    static_assert(2 * R <= 16 && K_OFF + 17 < W - 1, "a lane's residues are four words; the widest initial row fits");
    static_assert(PACK_REBASE + PACK_STEP_MAX + R * PACK_GE_MAX + (W - 1) * PACK_GE_MAX < 0x8000, "the values fit 16 bits");
    static_assert(PACK_REBASE - PACK_REBASE_BY - PACK_XMAX > PACK_STEP_MAX, "a dead cell stays dead after the origin's move");
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ uint2 tab[16];
    const int32_t ge = P->gap_extend, go = P->gap_open, goe = go + ge;
    if (threadIdx.x < 16) {
        uint32_t b[8];
        for (int c = 0; c < 8; ++c) {
            int32_t v = c < 4 ? P->matrix[threadIdx.x * 16 + c] : c == 4 ? P->matrix[threadIdx.x * 16 + 14] : -1000;
            v += 2 * ge;
            b[c] = (uint32_t)(v < -128 ? -128 : v) & 0xffu;
        }
        tab[threadIdx.x] = make_uint2(b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24, b[4] | b[5] << 8 | b[6] << 16 | b[7] << 24);
    }
    __syncthreads();
    if (n_dev) n_rec = *n_dev;
    if (list) n_rec = *n_list;
    const StreamDiv div_ge(ge);
    const int lane = threadIdx.x & 31, gl = lane & (G - 1);
    const unsigned gmask = (G == 32 ? FULL : ((1u << G) - 1u)) << (lane & ~(G - 1));
    const bool first_lane = gl == 0, last_lane = gl == G - 1;
    const int col0 = gl * 2 * R;  // this lane's first window diagonal
    const uint32_t half_base = pack2(ge * col0, ge * (col0 + R));

    uint32_t H[R], E[R], sel[R], S[R];  // S: the row of the best
#pragma unroll
    for (int r = 0; r < R; ++r) H[r] = E[r] = S[r] = 0, sel[r] = 0x8080u;
    // the extension, the same in all lanes of a group
    uint64_t item = 0, next_item = 0;
    uint32_t t = 0, cells = 0;
    bool idle = false, bail = false, need = true, running = false;
    const uint8_t *ap = nullptr, *bp = nullptr;  // the residues two rows on: the row's, the last diagonal's
    int32_t best = 0, best_bo = 0, best_k0 = 0;
    uint32_t best_a = 0;
    // best + origin, plain and as the packed start of the running best; both grow by 2 gap_extend a row
    int32_t bo = 0, step = 0;
    uint32_t pb = 0, step2 = 0;
    uint32_t neg_x = 0, base_x = 0;
    int32_t row = 0, kr = 0, left_rows = 0, k0 = 0;  // kr = k0 + row - columns; left_rows = rows - row
    uint32_t a_cur = 0, a_nx = 0, b_nx = 0x80u;

    auto take = [&]() -> uint64_t {  // by all lanes of a group
        uint32_t v = 0;
        if (first_lane) v = atomicAdd(queue, 1u);
        return __shfl_sync(gmask, v, 0, G);
    };
    next_item = take();

    int32_t lc = 0, fc = 0, fj = 0;
    uint32_t width = 0;
    bool slow = true, odd = false;
    for (;;) {
        if (__any_sync(FULL, slow)) {
            bool right = false, left = false;
            // what one lane saw holds for its group: the groups' lanes stay together
            const bool odd_group = (__ballot_sync(FULL, odd) & gmask) != 0;
            const bool slow_group = (__ballot_sync(FULL, slow) & gmask) != 0;
            if (slow_group && !need) {
                // the extension's end (gapped.rs:298-334), a record for the warp kernel, or a window move
                if (lc < 0) need = true;
                else if (fc == 0 || lc == W - 1) need = bail = true;
                else if (fj > 0 || left_rows <= 0) need = true;
                else if (width > window || cells > max_cells || odd_group) need = bail = true;
                else {
                    right = lc > W - 8 && fc > R + 4;
                    left = fc < 4 && lc < W - R - 8;
                }
                if (need) cells -= width;  // no next row
            }
            const bool rebase = !need && bo > PACK_REBASE;
            if (__any_sync(FULL, right || left || rebase)) {
                // moves of the window by R diagonals, of the origin.  The new diagonals' residues:
                // the last diagonal's next one is at bp - 1 before the move
                const uint32_t keep = last_lane ? 0u : FULL, keep_l = first_lane ? 0u : FULL;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t hd = __shfl_down_sync(FULL, H[r], 1, G) & keep, ed = __shfl_down_sync(FULL, E[r], 1, G) & keep;
                    const uint32_t sd = __shfl_down_sync(FULL, sel[r], 1, G);
                    const uint32_t hu = __shfl_up_sync(FULL, H[r], 1, G) & keep_l, eu = __shfl_up_sync(FULL, E[r], 1, G) & keep_l;
                    const uint32_t su = __shfl_up_sync(FULL, sel[r], 1, G);
                    if (right) {
                        H[r] = prmt(H[r], hd, 0x5432);
                        E[r] = prmt(E[r], ed, 0x5432);
                        const uint32_t nw = last_lane ? (uint32_t)bp[r - 1] : sd;
                        if (last_lane) odd |= pack_odd(nw) != 0;
                        sel[r] = prmt(sel[r], nw, 0x0041);
                    } else if (left) {
                        H[r] = prmt(hu, H[r], 0x5432);
                        E[r] = prmt(eu, E[r], 0x5432);
                        const uint32_t nw = first_lane ? (uint32_t)bp[r - 1 - W - R] : su >> 8;
                        if (first_lane) odd |= pack_odd(nw) != 0;
                        sel[r] = prmt(nw, sel[r], 0x0040);
                    }
                }
                if (right) {
                    k0 += R;
                    kr += R;
                    bp += R;
                    bo += ge * R;
                    pb += pack2(ge * R, ge * R);
                } else if (left) {
                    k0 -= R;
                    kr -= R;
                    bp -= R;
                    bo -= ge * R;
                    pb -= pack2(ge * R, ge * R);
                }
                if (right || left) b_nx = bp[-1];
                if (rebase) {
                    const uint32_t by = pack2(-PACK_REBASE_BY, -PACK_REBASE_BY);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        H[r] = __viaddmax_s16x2_relu(H[r], by, 0u);
                        E[r] = __viaddmax_s16x2_relu(E[r], by, 0u);
                    }
                    bo -= PACK_REBASE_BY;
                    pb -= pack2(PACK_REBASE_BY, PACK_REBASE_BY);
                }
                const bool moved_odd = (__ballot_sync(FULL, (right || left) && odd) & gmask) != 0;
                if (moved_odd) need = bail = true;
            }
            if (__any_sync(FULL, need && running)) {
                // the first window diagonal with the best, in the best's row
                const uint32_t goal = pack2(best_bo, best_bo) + half_base;
                uint32_t c = 1000;
#pragma unroll
                for (int r = R - 1; r >= 0; --r)
                    if (((S[r] ^ (goal + (0x80008000u - K.live[r]))) >> 16) == 0) c = col0 + R + r;
#pragma unroll
                for (int r = R - 1; r >= 0; --r)
                    if (((S[r] ^ (goal + (0x80008000u - K.live[r]))) & 0xffffu) == 0) c = col0 + r;
#pragma unroll
                for (int d = 1; d < G; d <<= 1) c = min(c, __shfl_xor_sync(FULL, c, d, G));
                if (need && running) {
                    const uint32_t b = best > 0 ? (uint32_t)((int32_t)c + best_k0 + (int32_t)best_a) : 0u;
                    if (first_lane) pack_store(out + t, (int)(item & 1u), PackSide{best, best_a, b, cells}, !bail);
                    running = bail = false;
                }
            }
            while (need && !idle) {
                item = next_item;
                if (item >= 2 * n_rec) {
                    idle = true;
                    // an idle group's rows stay dead
                    step = 0;
                    step2 = 0;
                    bo = PACK_REBASE_BY;
                    pb = pack2(bo, bo) + half_base;
                    neg_x = 0;
                    base_x = half_base;
#pragma unroll
                    for (int r = 0; r < R; ++r) H[r] = E[r] = 0;
                    break;
                }
                next_item = take();
                t = list ? list[item >> 1] : (uint32_t)(item >> 1);
                // start the extension (gapped.rs:165-200): the initial row's cells 0 .. J
                const uint4* gp = reinterpret_cast<const uint4*>(geo + t);
                const uint4 g0 = gp[0], g1 = gp[1];
                const int32_t X = (int32_t)reinterpret_cast<const uint32_t*>(geo + t)[10];
                ap = (const uint8_t*)(((uint64_t)g0.w << 32) | g0.z);
                bp = (const uint8_t*)(((uint64_t)g0.y << 32) | g0.x);
                int32_t rows = (int32_t)g1.w, nb = (int32_t)g1.z;
                if (!(item & 1u)) {
                    ap += K.s_stride + (g1.y - g1.w);
                    bp += K.q_stride + (g1.x - g1.z);
                } else {
                    ap += g1.w;
                    bp += g1.z;
                    rows = (int32_t)g1.y - rows;
                    nb = (int32_t)g1.x - nb;
                }
                if (rows <= 0 || nb <= 0) {  // an empty extension: score 0
                    if (first_lane) pack_store(out + t, (int)(item & 1u), PackSide{0, 0, 0, 0}, true);
                    continue;
                }
                const int32_t jmax = (int32_t)div_ge((uint32_t)(X - goe)) + 1;
                const int32_t J = jmax < nb ? jmax : nb;
                // this lane's residues: 2 R bytes from an unaligned address, in whole words
                const uint8_t* bl = bp + (col0 - K_OFF);
                const uint32_t* bw = reinterpret_cast<const uint32_t*>((uintptr_t)bl & ~(uintptr_t)3);
                const uint32_t sh = 8u * (uint32_t)((uintptr_t)bl & 3u);
                uint32_t w[5], v[4];
#pragma unroll
                for (int i = 0; i < 5; ++i) w[i] = bw[i];
                a_cur = ap[0];
                a_nx = ap[1];
                b_nx = bp[W - K_OFF];
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = __funnelshift_r(w[i], w[i + 1], sh);
                uint32_t od = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (2 * R > 4 * i) od |= pack_odd(v[i]) & (2 * R >= 4 * i + 4 ? 0xffffffffu : (1u << (8 * (2 * R - 4 * i))) - 1u);
                if (__any_sync(gmask, od != 0) || (uint32_t)J + 1 > window) {
                    if (first_lane) pack_store(out + t, (int)(item & 1u), PackSide{0, 0, 0, 0}, false);
                    continue;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int lo = r, hi = R + r;
                    sel[r] = prmt(v[lo / 4], v[hi / 4], (uint32_t)(lo % 4) | (uint32_t)(4 + hi % 4) << 4);
                }
                best = 0;
                best_a = 0;
                bo = X + 256;
                const int32_t base = bo + ge * K_OFF;
                step = 2 * ge;
                step2 = pack2(step, step);
                pb = pack2(bo, bo) + half_base;
                neg_x = pack2(-X, -X);
                base_x = half_base - pack2(X, X);
                k0 = -K_OFF;
                row = 0;
                kr = k0 - nb;
                left_rows = rows;
                cells = (uint32_t)J + 1;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int32_t ka = col0 + r - K_OFF, kb = ka + R;
                    // gap cells 1 .. J; cell J's diagonal leads out of the first row's band
                    const int32_t ea = ka > 0 && ka <= J ? base - 2 * go : 0, eb = kb > 0 && kb <= J ? base - 2 * go : 0;
                    E[r] = pack2(ea, eb);
                    H[r] = pack2(ka > 0 && ka < J ? base - go : 0, kb > 0 && kb < J ? base - go : 0);
                    if (ka == 0 || kb == 0) {
                        H[r] |= ka == 0 ? pack2(base, 0) : pack2(0, base);
                        E[r] |= ka == 0 ? pack2(base - go, 0) : pack2(0, base - go);
                    }
                }
                ap += 2;
                bp += W - K_OFF + 1;
                need = false;
                running = true;
            }
            __syncwarp();
            odd = false;
            if (!__any_sync(FULL, !idle)) break;
        }

        // ---- one row
        bo += step;
        pb += step2;
        ++row;
        ++kr;
        --left_rows;
        const uint2 tb = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(tab) + a_cur);
        uint32_t x = __shfl_down_sync(FULL, E[0], 1, G);
        if (last_lane) x = 0;
        const uint32_t e_edge = prmt(E[0], x, 0x5432);
        uint32_t f = 0, p = pb;
        uint32_t T[R], F[R], pr[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            T[r] = __viaddmax_s16x2(H[r], prmt(tb.x, tb.y, sel[r]), r + 1 < R ? E[r + 1 < R ? r + 1 : r] : e_edge);
            F[r] = f;
            f = __viaddmax_s16x2(T[r], K.neg_go, f);
            p = __viaddmax_s16x2(T[r], K.neg_ge[r], p);
            pr[r] = p;
        }
        // prefix maxima over the half-lanes: the gap in the low half, the running best in the high
        const uint32_t pg = p - half_base;
        const uint32_t u_lo = prmt(f, pg, 0x5410);
        uint32_t inc = __vmaxs2(u_lo, prmt(f, pg, 0x7632));
#pragma unroll
        for (int d = 1; d < G; d <<= 1) inc = __vmaxs2(inc, __shfl_up_sync(FULL, inc, d, G));
        uint32_t ex = __shfl_up_sync(FULL, inc, 1, G);
        if (first_lane) ex = pb << 16;
        const int32_t rb = (int32_t)(__shfl_sync(FULL, inc, G - 1, G) >> 16);
        const uint32_t ex_hi = __vmaxs2(ex, u_lo);
        const uint32_t f_in = prmt(ex, ex_hi, 0x5410), p_in = prmt(ex, ex_hi, 0x7632) + base_x;
        const bool better = rb > bo;
        uint32_t al = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t cell = r == 0 ? __vmaxs2(T[0], f_in) : __vimax3_s16x2(T[r], F[r], f_in);
            const uint32_t thr = __viaddmax_s16x2(pr[r], neg_x, p_in);
            const uint32_t live = prmt(cell + K.live[r] - thr, 0, 0xbb99);
            const uint32_t up = r + 1 < R ? E[r + 1 < R ? r + 1 : r] : e_edge;
            H[r] = cell & live;
            al |= live & (0x00010001u << r);
            E[r] = __viaddmax_s16x2(H[r], K.neg_go, up);
            if (better) S[r] = H[r];
        }
        // first and last live diagonal of the window
        const uint32_t bits = (al & 0xffffu) | (al >> 16 << R);
        uint32_t z = bits ? pack2(col0 + 31 - __clz((int)bits), 1 - col0 - __ffs((int)bits)) : pack2(-1000, -1000);
#pragma unroll
        for (int d = 1; d < G; d <<= 1) z = __vmaxs2(z, __shfl_xor_sync(FULL, z, d, G));
        lc = (int16_t)z;
        fc = -((int32_t)z >> 16);
        if (better) {
            best += rb - bo;
            pb += (uint32_t)(rb - bo) * 0x00010001u;
            bo = rb;
            best_bo = rb;
            best_k0 = k0;
            best_a = (uint32_t)row;
        }
        fj = fc + kr;  // the first live column, less the columns
        width = (uint32_t)(min(lc + kr + 2, 1) - fj);
        cells += width;
        // the residues one row on
        const uint32_t s0 = sel[0];
        uint32_t sn = __shfl_down_sync(FULL, s0, 1, G);
        if (last_lane) {
            sn = b_nx;
            odd = pack_odd(b_nx) != 0;
        }
#pragma unroll
        for (int r = 0; r + 1 < R; ++r) sel[r] = sel[r + 1];
        sel[R - 1] = prmt(s0, sn, 0x0041);
        a_cur = a_nx;
        if (!idle && left_rows > 0) {
            a_nx = *ap++;
            b_nx = *bp++;
        }
        slow = !idle && (max(max(max(lc - (W - 8), 4 - fc), max(fj, 1 - left_rows)), max(-lc, bo - PACK_REBASE)) > 0 ||
                         cells > max_cells || width > window || odd);
    }
}

// Joins k_prelim_pack's two extensions of each record (engine.rs:1380-1397); one with an extension
// that did not fit goes to `wide`.
__global__ void __launch_bounds__(256)
k_prelim_pack_join(uint64_t n_rec, const PrelimGeo* __restrict__ geo, PrelimOut* __restrict__ out, int32_t cutoff,
                   uint32_t* __restrict__ wide, unsigned int* __restrict__ n_wide,
                   unsigned long long* __restrict__ cells_total, uint32_t* __restrict__ cells_out,
                   const unsigned int* __restrict__ n_dev, const uint32_t* __restrict__ list,
                   const unsigned int* __restrict__ n_list) {
    if (n_dev) n_rec = *n_dev;
    if (list) n_rec = *n_list;
    unsigned long long cells = 0;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n_rec; k += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t t = list ? list[k] : (uint32_t)k;
        const uint16_t* ok = reinterpret_cast<const uint16_t*>(out + t) + 12;
        if (!ok[0] || !ok[1]) {
            wide[atomicAdd(n_wide, 1u)] = t;
            if (cells_out) cells_out[t] = 0xffffffffu;
            continue;
        }
        const PackSide l = pack_side(out + t, 0), r = pack_side(out + t, 1);
        PrelimOut o{INT32_MIN, 0, 0, 0, 0, 0, 0};
        const int32_t total = l.score + r.score;
        if (total >= 0 && total >= cutoff) {
            const uint4* gp = reinterpret_cast<const uint4*>(geo + t);
            const uint4 g1 = gp[1], g2 = gp[2];
            const uint32_t qa = g1.x, sa = g1.y, qp = g1.z, sp = g1.w;
            uint32_t q0 = qp - l.b, s0 = sp - l.a, q1 = qp + r.b, s1 = sp + r.a;
            if (!(g2.w & 1u)) {
                const uint32_t x0 = qa - q1, x1 = qa - q0, x2 = sa - s1, x3 = sa - s0;
                q0 = x0; q1 = x1; s0 = x2; s1 = x3;
            }
            o = PrelimOut{total, q0, q1, s0, s1, g2.x, g2.y};
        }
        out[t] = o;
        if (cells_out) cells_out[t] = l.cells + r.cells;
        cells += l.cells + r.cells;
    }
    for (int d = 16; d; d >>= 1) cells += __shfl_xor_sync(0xffffffffu, cells, d);
    if ((threadIdx.x & 31) == 0 && cells) atomicAdd(cells_total, cells);
}

}  // namespace rmb
