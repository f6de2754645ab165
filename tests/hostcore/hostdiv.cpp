// Host build of the batched launches' tile division (test harness only; csrc/planediv.cuh compiled with g++).
#include <cstdint>

#include "../../pyocean_b200/csrc/planediv.cuh"

extern "C" {

// Mismatches of tile_div(x, tile_magic(d, count), d) against x / d over 0 <= x < d count: every x where there are at most
// `all` of them, else those next to the first and last multiples of d and every step-th one.
long long check_tile_div(long long d, long long count, long long all)
{
    const long long total = d * count;
    const unsigned long long m = po::tile_magic(d, count);
    auto wrong = [&](long long x) { return x >= 0 && x < total && po::tile_div((int)x, m, (int)d) != (int)(x / d); };
    long long bad = 0;
    if (total <= all) {
        for (long long x = 0; x < total; ++x) bad += wrong(x);
        return bad;
    }
    const long long step = count / (all / 8) + 1;
    for (long long q = 0; q <= count; q += q < 1000 || q + 1000 > count ? 1 : step)
        for (long long e = -2; e <= 2; ++e) bad += wrong(q * d + e);
    return bad;
}

}  // extern "C"
