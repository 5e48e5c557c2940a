// Host build of the sequential DUST pass (rmb_dust.cuh) for tests/test_dust_segments.py.
#include <vector>

#include "../rmblast_b200/csrc/rmb_dust.cuh"

extern "C" int dust_host(const uint8_t* bases, uint32_t n, uint8_t* out) {
    std::vector<rmb::DustPerfect> scratch(rmb::DUST_PERFECT_CAP);
    return rmb::dust_query(bases, n, out, scratch.data()) ? 0 : 1;
}
