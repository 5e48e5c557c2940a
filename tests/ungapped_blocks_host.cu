// Host build of UngBlocks (rmb_ungapped.cuh, the walk of k_ungapped, k_dedup_extend and k_bucket_dedup)
// checked against the oracle's extension on seeded random hits.
//
//   ungapped_blocks_host <hits> <seed> <xdrop> <matrix>
//
// Prints one line: "hits N bad B steps S".  Sequences lie at every offset from an aligned word, the
// bytes around them are no sequence's; seeds reach both ends; odd codes and score tables with large entries.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../oracle/rmb_oracle.hpp"
#include "../rmblast_b200/csrc/rmb_ungapped.cuh"

int main(int argc, char** argv) {
    if (argc < 5) {
        fprintf(stderr, "usage: ungapped_blocks_host hits seed xdrop matrix\n");
        return 2;
    }
    const int n = atoi(argv[1]);
    std::mt19937_64 rng((uint64_t)atoll(argv[2]));
    const int xdrop = atoi(argv[3]);
    rmbo::Matrix mat = rmbo::load_matrix(argv[4]);
    int bad = 0;
    unsigned long long steps = 0;
    for (int k = 0; k < n; ++k) {
        if (k % 4 == 3) mat.s[rng() % 15][rng() % 15] = (int32_t)(rng() % 4001) - 2000;  // asymmetric, large
        if (k % 64 == 0) mat = rmbo::load_matrix(argv[4]);
        int32_t flat[256], tab[256];
        for (int a = 0; a < 16; ++a)
            for (int b = 0; b < 16; ++b) flat[a * 16 + b] = mat.s[a][b];
        for (int i = 0; i < 256; ++i) tab[rmb::ung_slot(i)] = rmb::ung_entry(i, flat);
        const bool tiny = k % 3 == 0;
        const int sl = 1 + (int)(rng() % (tiny ? 40 : 3000)), ql = 1 + (int)(rng() % (tiny ? 40 : 3000));
        const size_t qat = rng() % 8, sat = rng() % 8;  // where the wrapped sequences start in their first word
        std::vector<uint2> qmem((qat + ql + 2) / 8 + 1), smem((sat + sl + 2) / 8 + 1);
        uint8_t *qw = (uint8_t*)qmem.data() + qat, *sw = (uint8_t*)smem.data() + sat;
        for (size_t j = 0; j < qmem.size() * 8; ++j) ((uint8_t*)qmem.data())[j] = (uint8_t)(rng() % 15);
        for (size_t j = 0; j < smem.size() * 8; ++j) ((uint8_t*)smem.data())[j] = (uint8_t)(rng() % 15);
        qw[0] = qw[ql + 1] = sw[0] = sw[sl + 1] = 15;
        for (int j = 1; j <= sl; ++j) sw[j] = (uint8_t)(rng() % 4);
        for (int j = 1; j <= ql; ++j) qw[j] = (uint8_t)(rng() % 4);
        const int seg = 1 + (int)(rng() % std::min(sl, ql));
        const int s0 = (int)(rng() % (sl - seg + 1)), q0 = (int)(rng() % (ql - seg + 1));
        const int div = (int)(rng() % 30);
        for (int j = 1; j <= seg; ++j)
            if ((int)(rng() % 100) >= div) qw[q0 + j] = sw[s0 + j];
        for (int j = 1; j <= ql; ++j)
            if (rng() % 300 == 0) qw[j] = (uint8_t)(4 + rng() % 11);
        const int at = k % 5 == 0 ? 0 : k % 5 == 1 ? seg - 1 : (int)(rng() % seg);
        const int qo = q0 + at, so = s0 + at;
        const rmbo::UngappedResult want =
            rmbo::extend_ungapped(qw, ql + 2, sw, sl + 2, (uint32_t)qo, (uint32_t)so, mat, xdrop);
        rmb::UngBlocks w;
        w.start(qw, sw, ql, sl, qo, so, xdrop);
        do ++steps;
        while (!w.step(tab));
        int32_t sc;
        uint32_t a, b, c, d;
        w.result(sc, a, b, c, d);
        if (sc != want.score || a != want.q_start || b != want.q_end || c != want.s_start || d != want.s_end) {
            if (bad < 5)
                fprintf(stderr, "hit %d: want %d %u-%u %u-%u got %d %u-%u %u-%u\n", k, want.score, want.q_start,
                        want.q_end, want.s_start, want.s_end, sc, a, b, c, d);
            ++bad;
        }
    }
    printf("hits %d bad %d steps %llu\n", n, bad, steps);
    return bad != 0;
}
