#pragma once
// Traceback X-drop DP with a row's band in registers and the trace walk (the body of
// k_traceback_pack): search/gapped.rs:450-757 align_ex + traceback_flat, one extension a warp.
//
// The rows are k_prelim_pack's (rmb_prelim_pack.cuh: window of diagonals, packed 16-bit values,
// coordinates, exactness), with the whole warp on one extension, TB_W = 128 diagonals, four a lane.  The
// scores are 16-bit table entries (two byte lookups and a merge), so the X-drop is limited by the
// window alone, and the scores by what keeps a dead cell dead (TB_LIVE).  They hold the bases and N; a
// column of another ambiguity code looks its score up in shared memory.  A cell's trace is four bits:
// the vertical gap beat the diagonal, the horizontal gap beat both, and either gap's extension is at
// least its opening, gapped.rs:577-618's op byte; a row's 128 are 64 bytes, one 16-bit store a lane,
// with the row's window position beside them.  On cells below the X-drop threshold they may differ
// from the reference's, and no path visits those.
//
// The walk goes by runs: lane l looks at the cell l steps up the path's diagonal, and the warp takes the
// run of substitutions to the first gap, 32 at most, at once; a gap's cells go one by one.
//
// Bound: latency.  A launch has few, long alignments, and a row waits for the one before: two
// prefix-maximum scans of five shuffles in one, two reductions and the row's 30 packed operations.
#include "rmb_prelim_pack.cuh"

namespace rmb {

constexpr int TB_R = 2, TB_W = 64 * TB_R, TB_K = TB_W / 2 - 2;
constexpr uint32_t TB_ROW_BYTES = TB_W / 2 + 4;  // trace and window position of a row
constexpr int32_t TB_SCORE_MIN = -8192;          // a blocked column's score: ends any path
constexpr int32_t TB_LIVE = 256;                 // live values stay above it: no score of a cell reaches it
constexpr int32_t TB_GE_MAX = 40, TB_XMAX = 4000;
static_assert(PACK_REBASE + TB_LIVE + (2 + 2 * TB_R) * TB_GE_MAX + (TB_W - 1) * TB_GE_MAX < 0x8000, "the values fit 16 bits");
static_assert(PACK_REBASE - PACK_REBASE_BY - TB_XMAX > TB_LIVE + 2 * TB_GE_MAX, "a dead cell stays dead after the origin's move");
static_assert(-TB_SCORE_MIN > TB_XMAX + 2 * TB_GE_MAX, "a blocked column ends any path");

// Status of an extension that its window does not fit: the byte-trace kernel takes it.
constexpr int TB_WIDE = 4;

struct TbTable {  // scores with both gap decays: row residue x code, low and high bytes of codes 0-3, 4-7
    uint4 row[16];
    int16_t all[256];  // the same for every pair of residues
};

__device__ __forceinline__ uint32_t tb_code(uint32_t base) { return base < 4 ? base : base == 14 ? 4u : 6u; }

// One extension: row residues a[dir * i], i < m, column residues b[dir * j], j < n.  Returns 0 ok, 2 the
// trace rows or the script's slot ran out, 3 the walk did not reach the origin, TB_WIDE.
__device__ __forceinline__ int tb_pack_extend(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b, int dir,
                                              int32_t m, int32_t n, int32_t go, int32_t ge, int32_t xdrop,
                                              const TbTable& tab, uint16_t* trace, int32_t* win, uint32_t rows_cap,
                                              int32_t& score_out, uint32_t& a_len, uint32_t& b_len, uint32_t* ops_rev,
                                              uint32_t ops_cap, uint32_t& n_ops, uint64_t& cells) {
    constexpr int R = TB_R, W = TB_W;
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    score_out = 0;
    a_len = b_len = 0;
    n_ops = 0;
    if (m <= 0 || n <= 0) return 0;
    const int32_t goe = go + ge, X = xdrop > goe ? xdrop : goe;
    const int32_t jmax = (X - goe) / ge + 1, J = jmax < n ? jmax : n;
    const int col0 = lane * 2 * R;
    const uint32_t half_base = pack2(ge * col0, ge * (col0 + R));
    const uint32_t neg_go = pack2(-go, -go), neg_x = pack2(-X, -X), base_x = half_base - pack2(X, X);
    const uint32_t step2 = pack2(2 * ge, 2 * ge);
    auto code_at = [&](int32_t j) -> uint32_t { return j < 0 ? 0u : j >= n ? 5u : tb_code(b[(ptrdiff_t)dir * j]); };

    uint32_t H[R], E[R], sel[R], S[R];
    int32_t bo = X + TB_LIVE, k0 = -TB_K, best = 0, best_bo = 0, best_k0 = 0, row = 0;
    uint32_t best_a = 0;
    cells = (uint64_t)J + 1;
    bool odd = false;
    {
        const int32_t base = bo + ge * TB_K;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int32_t ka = col0 + r - TB_K, kb = ka + R;
            const int32_t ea = ka < 0 || ka > J ? 0 : ka == 0 ? base - go : base - 2 * go;
            const int32_t eb = kb < 0 || kb > J ? 0 : kb == 0 ? base - go : base - 2 * go;
            E[r] = pack2(ea, eb);
            // cell J's diagonal leads out of the first row's band
            H[r] = pack2(ea && ka != J ? ea + go : 0, eb && kb != J ? eb + go : 0);
            const uint32_t ca = code_at(ka), cb = code_at(kb);
            odd |= ca == 6 || cb == 6;
            sel[r] = ca | cb << 8;
            S[r] = 0;
        }
    }
    bool codes = __any_sync(FULL, odd);  // some column of the window has code 6
    uint32_t pb = pack2(bo, bo) + half_base;
    uint32_t a_cur = a[0] & 15u, a_nx = m > 1 ? a[dir] & 15u : 0u;
    uint32_t b_nx = code_at(W - TB_K);  // the last diagonal's code in the second row
    for (;;) {
        if ((uint32_t)row >= rows_cap) return 2;
        bo += 2 * ge;
        pb += step2;
        const uint4 tb = tab.row[a_cur];
        uint32_t x = __shfl_down_sync(FULL, E[0], 1);
        if (lane == 31) x = 0;
        const uint32_t e_edge = prmt(E[0], x, 0x5432);
        uint32_t f = 0, p = pb, D[R], T[R], F[R], pr[R], sc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) sc[r] = prmt(prmt(tb.x, tb.y, sel[r]), prmt(tb.z, tb.w, sel[r]), 0x6240);
        // Code 6, an ambiguity code other than N: the residue's own score, while the window has one.  (Such
        // extensions went to k_traceback_warp before: 40 queries of 60 kb against 500 consensi with 0.05 % of such
        // codes 28.5 ms, 9.2 now, with 1 % 28.6 and 12.9.)
        if (codes) {
            bool some = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int32_t j = col0 + r + k0 + row;
                if ((sel[r] & 0xffu) == 6) {
                    sc[r] = (sc[r] & 0xffff0000u) | (uint16_t)tab.all[a_cur * 16 + (b[(ptrdiff_t)dir * j] & 15u)];
                    some = true;
                }
                if ((sel[r] >> 8 & 0xffu) == 6) {
                    sc[r] = (sc[r] & 0xffffu) | (uint32_t)(uint16_t)tab.all[a_cur * 16 + (b[(ptrdiff_t)dir * (j + R)] & 15u)] << 16;
                    some = true;
                }
            }
            codes = __any_sync(FULL, some);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            D[r] = __viaddmax_s16x2_relu(H[r], sc[r], 0u);
            T[r] = __vmaxs2(D[r], r + 1 < R ? E[r + 1 < R ? r + 1 : r] : e_edge);
            F[r] = f;
            f = __viaddmax_s16x2(T[r], neg_go, f);
            p = __viaddmax_s16x2(T[r], pack2(-ge * r, -ge * r), p);
            pr[r] = p;
        }
        const uint32_t pg = p - half_base;
        const uint32_t u_lo = prmt(f, pg, 0x5410);
        uint32_t inc = __vmaxs2(u_lo, prmt(f, pg, 0x7632));
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) inc = __vmaxs2(inc, __shfl_up_sync(FULL, inc, d));
        uint32_t ex = __shfl_up_sync(FULL, inc, 1);
        if (lane == 0) ex = pb << 16;
        const int32_t rb = (int32_t)(__shfl_sync(FULL, inc, 31) >> 16);
        const uint32_t ex_hi = __vmaxs2(ex, u_lo);
        const uint32_t f_in = prmt(ex, ex_hi, 0x5410), p_in = prmt(ex, ex_hi, 0x7632) + base_x;
        const bool better = rb > bo;
        uint32_t tr[R];
        int32_t last = -1, first = W;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t fv = __vmaxs2(F[r], f_in);
            const uint32_t cell = __vmaxs2(T[r], fv);
            const uint32_t thr = __viaddmax_s16x2(pr[r], neg_x, p_in);
            const uint32_t live = prmt(cell + (0x80008000u - (uint32_t)(ge * r) * 0x00010001u) - thr, 0, 0xbb99);
            const uint32_t up = r + 1 < R ? E[r + 1 < R ? r + 1 : r] : e_edge;
            H[r] = cell & live;
            const uint32_t open = __viaddmax_s16x2_relu(H[r], neg_go, 0u);
            const uint32_t c1 = up + 0x7fff7fffu - D[r], c2 = fv + 0x7fff7fffu - T[r];
            const uint32_t c3 = up + 0x80008000u - open, c4 = fv + 0x80008000u - open;
            tr[r] = (c1 & 0x80008000u) | ((c2 >> 1) & 0x40004000u) | ((c3 >> 2) & 0x20002000u) | ((c4 >> 3) & 0x10001000u);
            E[r] = __vmaxs2(open, up);
            if (better) S[r] = H[r];
            // columns in the order of lo 0, lo 1, hi 0, hi 1
            if (live & 0xffffu) {
                last = max(last, col0 + r);
                first = min(first, col0 + r);
            }
            if (live >> 16) {
                last = max(last, col0 + R + r);
                first = min(first, col0 + R + r);
            }
        }
        {
            const uint32_t y = ((tr[0] >> 12) & 0x000f000fu) | ((tr[1] >> 8) & 0x00f000f0u);
            trace[(uint64_t)row * 32 + lane] = (uint16_t)prmt(y, 0, 0x4420);
            if (lane == 0) win[row] = k0;
        }
        const int32_t lc = __reduce_max_sync(FULL, last), fc = __reduce_min_sync(FULL, first);
        ++row;
        if (better) {
            best += rb - bo;
            pb += (uint32_t)(rb - bo) * 0x00010001u;
            bo = rb;
            best_bo = rb;
            best_k0 = k0;
            best_a = (uint32_t)row;
        }
        if (lc < 0) break;                           // nothing live
        if (fc == 0 || lc == W - 1) return TB_WIDE;  // a cell may have left the window
        const int32_t fj = fc + k0 + row;
        if (fj > n || row >= m) break;
        cells += (uint64_t)(min(lc + k0 + row + 2, n + 1) - fj);
        // the residues one row on
        {
            const uint32_t s0 = sel[0];
            uint32_t sn = __shfl_down_sync(FULL, s0, 1);
            if (lane == 31) sn = b_nx;
            codes |= __any_sync(FULL, lane == 31 && b_nx == 6) != 0;
#pragma unroll
            for (int r = 0; r + 1 < R; ++r) sel[r] = sel[r + 1];
            sel[R - 1] = prmt(s0, sn, 0x0041);
            a_cur = a_nx;
            a_nx = row + 1 < m ? a[(ptrdiff_t)dir * (row + 1)] & 15u : 0u;
            if (lane == 31) b_nx = code_at(W + k0 + row);
        }
        // the band in the middle, with room for a new best's gap to the right (36 diagonals at an X-drop of
        // 200); a band almost as wide as the window only from its edges
        const bool right = (lc > W - 28 && fc > 28) || (lc > W - 8 && fc > 8);
        const bool left = !right && ((fc < 20 && lc < W - 32) || (fc < 5 && lc < W - 14));
        if (right || left) {
            // the window a lane (2 R diagonals) along
            const int32_t by = right ? 2 * R : -2 * R;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint32_t hd = __shfl_down_sync(FULL, H[r], 1), ed = __shfl_down_sync(FULL, E[r], 1);
                const uint32_t hu = __shfl_up_sync(FULL, H[r], 1), eu = __shfl_up_sync(FULL, E[r], 1);
                const uint32_t sd = __shfl_down_sync(FULL, sel[r], 1), su = __shfl_up_sync(FULL, sel[r], 1);
                H[r] = right ? hd : hu;
                E[r] = right ? ed : eu;
                sel[r] = right ? sd : su;
                if (lane == (right ? 31 : 0)) {
                    H[r] = E[r] = 0;
                    const uint32_t ca = code_at(col0 + r + k0 + by + row), cb = code_at(col0 + R + r + k0 + by + row);
                    odd |= ca == 6 || cb == 6;
                    sel[r] = ca | cb << 8;
                }
            }
            k0 += by;
            bo += ge * by;
            pb += (uint32_t)(ge * by) * 0x00010001u;
            if (lane == 31) b_nx = code_at(W + k0 + row);
            codes |= __any_sync(FULL, odd) != 0;
            odd = false;
        }
        if (bo > PACK_REBASE) {
            const uint32_t by = pack2(-PACK_REBASE_BY, -PACK_REBASE_BY);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                H[r] = __viaddmax_s16x2_relu(H[r], by, 0u);
                E[r] = __viaddmax_s16x2_relu(E[r], by, 0u);
            }
            bo -= PACK_REBASE_BY;
            pb -= pack2(PACK_REBASE_BY, PACK_REBASE_BY);
        }
    }
    score_out = best;
    if (best == 0) return 0;
    {
        // the first window diagonal with the best, in the best's row
        const uint32_t goal = pack2(best_bo, best_bo) + half_base;
        uint32_t c = 1000;
#pragma unroll
        for (int r = R - 1; r >= 0; --r)
            if (((S[r] ^ (goal + (uint32_t)(ge * r) * 0x00010001u)) >> 16) == 0) c = col0 + R + r;
#pragma unroll
        for (int r = R - 1; r >= 0; --r)
            if (((S[r] ^ (goal + (uint32_t)(ge * r) * 0x00010001u)) & 0xffffu) == 0) c = col0 + r;
        c = __reduce_min_sync(FULL, c);
        a_len = best_a;
        b_len = (uint32_t)((int32_t)c + best_k0 + (int32_t)best_a);
    }
    __syncwarp();  // the rows' traces before the walk reads them
    int32_t aa = (int32_t)a_len, bq = (int32_t)b_len;
    int prev = 0;  // 0 substitution, 1 gap in a (horizontal), 2 gap in b (vertical)
    uint32_t cur_op = 0xffffffffu, cur_n = 0, nops = 0;
    for (uint32_t steps = a_len + b_len; aa > 0 || bq > 0;) {
        // lane l: the trace of the cell (aa - l, bq - l); from row 0 on a horizontal gap
        uint32_t raw = 4;
        const int32_t r = aa - 1 - lane;
        if (r >= 0) {
            const int32_t c = bq - aa - win[r];
            if (c >= 0 && c < W) raw = (trace[(uint64_t)r * 32 + (c >> 2)] >> (4 * (c & 3))) & 15u;
        }
        const int plain = raw & 4u ? 1 : raw & 8u ? 2 : 0;
        // a run of substitutions from here, or this cell's step
        const unsigned other = __ballot_sync(FULL, plain != 0);
        const uint32_t raw0 = __shfl_sync(FULL, raw, 0);
        const int plain0 = raw0 & 4u ? 1 : raw0 & 8u ? 2 : 0;
        int op = prev == 1 ? (raw0 & 1u ? 1 : plain0) : prev == 2 ? (raw0 & 2u ? 2 : plain0) : plain0;
        uint32_t len = 1;
        if (op == 0 && plain0 == 0) len = other ? (uint32_t)__ffs((int)other) - 1u : 32u;
        if (steps < len) return 3;
        steps -= len;
        prev = op;
        if (op != 1) aa = max(aa - (int32_t)len, 0);
        if (op != 2) bq = max(bq - (int32_t)len, 0);
        if ((uint32_t)op == cur_op) {
            cur_n += len;
        } else {
            if (cur_n) {
                if (nops >= ops_cap) return 2;
                if (lane == 0) ops_rev[nops] = (cur_op << 30) | cur_n;
                ++nops;
            }
            cur_op = (uint32_t)op;
            cur_n = len;
        }
    }
    if (cur_n) {
        if (nops >= ops_cap) return 2;
        if (lane == 0) ops_rev[nops] = (cur_op << 30) | cur_n;
        ++nops;
    }
    n_ops = nops;
    return 0;
}

}  // namespace rmb
