// Host check of the reciprocal's error bound (rcp_from, lare_div.cuh): from any
// seed within 2^-14 of 1/d the result is RN(1/d), and two of its three steps
// leave at most one ulp.
#include <cstdint>
#include <cstdio>
#include <random>

#include "lare_div.cuh"

using namespace sams::dev;

int main()
{
    std::mt19937_64 rng(29);
    long long bad = 0, coarse = 0;
    for (int t = 0; t < 3000000; ++t) {
        const uint64_t m = t % 3 == 0 ? 0xfffffffffffffull ^ (1ull << (rng() % 52)) : rng() & 0xfffffffffffffull;
        const uint64_t u = ((uint64_t)(1023 - 100 + (int)(rng() % 200)) << 52) | m;
        double d;
        std::memcpy(&d, &u, sizeof d);
        const double want = 1.0 / d;
        // an error of either sign, from nothing to the whole bound
        const double rel = (double)((int64_t)(rng() % 32769) - 16384) * 0x1p-28;
        const double seed = want + want * rel;
        if (rcp_from(d, seed) != want) ++bad;
        const double two = newton(d, newton(d, seed));
        if (two != want && two != std::nextafter(want, 0.0) && two != std::nextafter(want, 2 * want)) ++coarse;
    }
    std::printf("{\"bad\": %lld, \"coarse\": %lld}\n", bad, coarse);
    return bad || coarse ? 1 : 0;
}
