#pragma once
// The ungapped X-drop extension of one word hit (search/ungapped.rs:38-121) as a resumable walk:
// the left walk from the seed, then the right walk.  UngWalk is its plain form, one base a step; UngBlocks
// the kernels' form, eight bases a step.  Both compile for the host too, where the tests check them against
// the oracle's extension.
#include <cstdint>

namespace rmb {

struct UngWalk {
    const uint8_t* qb = nullptr;  // sentinel-wrapped query in the walk's strand frame (base q at qb[1 + q])
    const uint8_t* sb = nullptr;  // sentinel-wrapped plus-strand subject
    int32_t q = 0, s = 0, qlim = 0, slim = 0, dir = -1;
    int32_t sum = 0, score = 0, x = 0, xc = 0, best = 0, q_beg = 0;
    int32_t wq = 0, wsx = 0, qlen = 0, slen = 0;

    // From the seed (wq, wsx) with X-drop xdrop: the left walk first.
    __host__ __device__ __forceinline__ void start(const uint8_t* query, const uint8_t* subject, int32_t query_len,
                                                   int32_t subject_len, int32_t seed_q, int32_t seed_s, int32_t xdrop) {
        qb = query;
        sb = subject;
        qlen = query_len;
        slen = subject_len;
        wq = seed_q;
        wsx = seed_s;
        x = -xdrop;
        q = wq - 1; s = wsx - 1; dir = -1; qlim = -1; slim = -1;
        sum = 0; score = 0; xc = x; best = wq;
    }

    // One base: the walk's step on query base a and subject base c at (q, s), or its end when
    // at_end (q or s at its limit).  Returns 0 while walking, 1 when the left walk ended (the
    // right one starts at the seed), 2 when the right walk ended (the extension is done).
    __host__ __device__ __forceinline__ int on_base(bool at_end, uint8_t a, uint8_t c, const int32_t* mat) {
        bool stop = at_end;
        if (!stop) {
            if (a == 15 || c == 15) {
                stop = true;
            } else {
                sum += mat[((a & 15) << 4) | (c & 15)];
                if (sum > 0) {
                    best = dir < 0 ? q : q + 1;
                    score += sum;
                    if (dir > 0) xc = -score > x ? -score : x;
                    sum = 0;
                } else if (sum < xc) {
                    stop = true;
                }
            }
        }
        if (!stop) {
            q += dir;
            s += dir;
            return 0;
        }
        if (dir < 0) {
            q_beg = best;
            q = wq; s = wsx; dir = 1; qlim = qlen; slim = slen;
            sum = 0; xc = x; best = wq;
            return 1;
        }
        return 2;
    }

    // One base, as on_base.
    __host__ __device__ __forceinline__ int step(const int32_t* mat) {
        const bool end = q == qlim || s == slim;
        return on_base(end, end ? (uint8_t)15 : qb[1 + q], end ? (uint8_t)15 : sb[1 + s], mat);
    }

    // After step() returned 2: the extension in the walk's frame.
    __host__ __device__ __forceinline__ void result(int32_t& sc, uint32_t& q0, uint32_t& q1, uint32_t& s0,
                                                    uint32_t& s1) const {
        sc = score;
        q0 = (uint32_t)q_beg;
        q1 = (uint32_t)best;
        s0 = (uint32_t)(wsx - (wq - q_beg));
        s1 = (uint32_t)(wsx + (best - wq));
    }
};

#ifdef __CUDACC__
__host__ __device__ __forceinline__ uint2 ung_load(const uint2* p) {
#ifdef __CUDA_ARCH__
    return __ldg(p);
#else
    return *p;
#endif
}
__host__ __device__ __forceinline__ uint32_t ung_bytes(uint32_t lo, uint32_t hi, uint32_t sel) {  // __byte_perm
#ifdef __CUDA_ARCH__
    return __byte_perm(lo, hi, sel);
#else
    const uint64_t w = lo | (uint64_t)hi << 32;
    uint32_t r = 0;
    for (int k = 0; k < 4; ++k) r |= (uint32_t)(w >> 8 * (sel >> 4 * k & 7u) & 0xffu) << 8 * k;
    return r;
#endif
}
__host__ __device__ __forceinline__ uint32_t ung_shift(uint32_t lo, uint32_t hi, uint32_t by) {  // __funnelshift_r
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, by);
#else
    return (uint32_t)((lo | (uint64_t)hi << 32) >> (by & 31u));
#endif
}

// The walks' score table: entry ung_slot(16 a + c) for query code a, subject code c, so that in shared
// memory the 16 pairs of bases lie in 16 banks; a code 15 on either side (a sequence's end) ends any walk.
constexpr int32_t UNG_END = -(1 << 30), UNG_XMAX = 1 << 29;  // (an X-drop past it is out of any walk's reach)
__host__ __device__ __forceinline__ int ung_slot(int i) { return i ^ ((i >> 4 & 2) << 1); }
__host__ __device__ __forceinline__ int32_t ung_entry(int i, const int32_t* matrix) {
    return i >> 4 == 15 || (i & 15) == 15 ? UNG_END : matrix[i];
}
__device__ __forceinline__ void ung_table(int32_t* tab, const int32_t* __restrict__ matrix) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) tab[ung_slot(i)] = ung_entry(i, matrix);
}

// UngWalk eight bases a step.  A step's codes are two aligned words a sequence, one of them kept from
// the step before and the other asked for a step ahead, turned round on the left walk; the limits are
// the sentinels' scores.  Bound: one base a load (UngWalk) keeps the load unit busy with 32 lines a
// warp load, two of them a base; by words it is a quarter of a line a base, and the rest is
// arithmetic, about 14 operations a base.  Measured (B200), UngWalk and this: the walks of 75 M word hits
// of 1,000 contigs 26.4 -> 15.7 ms, the fused dedup of 500 consensi against each other 36 -> 19.
struct UngBlocks {
    struct Side {
        const uint2 *at, *last;  // the next word to ask for; the word of the walk's end
        uint2 cur, next;
        uint32_t shift;          // bits of cur that the walk has passed
    };
    Side a, c;
    const uint8_t *qb, *sb;
    int32_t wq, wsx, qlen, slen;
    int32_t x, xc, sum, score, n, best, q_beg;  // n: bases walked; best: of them, up to the best sum
    bool left;

    __host__ __device__ __forceinline__ uint2 word(const uint2* p) const {
        const uint2 w = ung_load(p);
        const uint32_t s0 = left ? 0x4567u : 0x3210u, s1 = left ? 0x0123u : 0x7654u;
        return make_uint2(ung_bytes(w.x, w.y, s0), ung_bytes(w.x, w.y, s1));
    }
    __host__ __device__ __forceinline__ const uint2* after(const Side& s) const {  // stays at the walk's end
        return s.at == s.last ? s.at : left ? s.at - 1 : s.at + 1;
    }
    __host__ __device__ __forceinline__ void enter(Side& s, const uint8_t* seq, int32_t len, int32_t i) {
        const uint64_t p = (uint64_t)(seq + 1 + i);
        s.last = (const uint2*)((uint64_t)(left ? seq : seq + 1 + len) & ~7ull);
        s.at = (const uint2*)(p & ~7ull);
        s.shift = 8u * (left ? 7u - (uint32_t)(p & 7u) : (uint32_t)(p & 7u));
        s.cur = word(s.at);
        s.at = after(s);
        s.next = word(s.at);
        s.at = after(s);
    }
    __host__ __device__ __forceinline__ uint2 codes(Side& s) {
        const bool high = s.shift >= 32;
        const uint32_t w0 = high ? s.cur.y : s.cur.x, w1 = high ? s.next.x : s.cur.y, w2 = high ? s.next.y : s.next.x;
        s.cur = s.next;
        s.next = word(s.at);
        s.at = after(s);
        return make_uint2(ung_shift(w0, w1, s.shift & 31u), ung_shift(w1, w2, s.shift & 31u));
    }
    // From the seed (wq, wsx) with X-drop xdrop: the left walk first.
    __host__ __device__ __forceinline__ void start(const uint8_t* query, const uint8_t* subject, int32_t query_len,
                                                   int32_t subject_len, int32_t seed_q, int32_t seed_s, int32_t xdrop) {
        qb = query;
        sb = subject;
        qlen = query_len;
        slen = subject_len;
        wq = seed_q;
        wsx = seed_s;
        x = xc = -min(xdrop, UNG_XMAX);
        sum = score = n = best = 0;
        left = true;
        enter(a, qb, qlen, wq - 1);
        enter(c, sb, slen, wsx - 1);
    }
    // Up to eight bases; true when the right walk has ended.
    __host__ __device__ __forceinline__ bool step(const int32_t* tab) {
        const uint2 qa = codes(a), sc = codes(c);
        bool run = true;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t q = h ? qa.y : qa.x;
            const uint32_t v = (q << 4 | (h ? sc.y : sc.x)) ^ ((q << 1) & 0x04040404u);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int32_t t = sum + tab[(v >> (8 * k)) & 0xffu];
                const bool up = run && t > 0;
                if (run) sum = min(t, 0);
                if (up) {
                    score += t;
                    best = n + 4 * h + k + 1;
                    if (!left) xc = max(-score, x);
                }
                run = run && t >= xc;
            }
        }
        n += 8;
        if (run) return false;
        if (!left) return true;
        q_beg = wq - best;
        left = false;
        xc = x;
        sum = n = best = 0;
        enter(a, qb, qlen, wq);
        enter(c, sb, slen, wsx);
        return false;
    }
    // After step() returned true: the extension in the walk's frame.
    __host__ __device__ __forceinline__ void result(int32_t& sc, uint32_t& q0, uint32_t& q1, uint32_t& s0,
                                                    uint32_t& s1) const {
        sc = score;
        q0 = (uint32_t)q_beg;
        q1 = (uint32_t)(wq + best);
        s0 = (uint32_t)(wsx - (wq - q_beg));
        s1 = (uint32_t)(wsx + best);
    }
};
#endif

}  // namespace rmb
