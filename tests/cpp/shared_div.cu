// Host check of the branch-free division (lare_div.cuh): where its conditions
// hold, rcp_fast and quot_check give the bits of the IEEE reciprocal and
// quotient, for random operands of every exponent, quotients next to rounding
// boundaries, denominators with few or nearly all bits set and special values.
#include <cfloat>
#include <cstdint>
#include <cstdio>
#include <random>

#include "lare_div.cuh"

using namespace sams::dev;

static long long bad = 0, used = 0;
static uint64_t bits(double x)
{
    uint64_t u;
    std::memcpy(&u, &x, sizeof u);
    return u;
}
static double real(uint64_t u)
{
    double x;
    std::memcpy(&x, &u, sizeof x);
    return x;
}
static void check(double x, double d)
{
    if (!plain_divisor(d)) return;
    const Rcp R = rcp_of(d);
    if (bits(R.r) != bits(1.0 / d)) ++bad;
    bool off = false;
    const double q = quot_check(x, R, off);
    if (off) {
        // only what is out of range may be refused
        const double w = std::fabs(x / d);
        if (w > 0x1p-599 && w < 0x1p599) ++bad;
        return;
    }
    ++used;
    if (bits(q) != bits(x / d)) ++bad;
}

int main()
{
    std::mt19937_64 rng(11);
    auto mantissa = [&] { return rng() & 0xfffffffffffffull; };
    auto with_exp = [&](int lo, int hi) {
        const uint64_t e = (uint64_t)(1023 + lo + (int)(rng() % (uint64_t)(hi - lo + 1)));
        return real((rng() & 0x8000000000000000ull) | (e << 52) | mantissa());
    };
    auto positive = [&](int lo, int hi) { return std::fabs(with_exp(lo, hi)); };
    for (int t = 0; t < 4000000; ++t) check(with_exp(-30, 30), positive(-30, 30));
    for (int t = 0; t < 2000000; ++t) check(with_exp(-1022, 1023), positive(-1022, 1023));
    for (int t = 0; t < 2000000; ++t) {  // x next to d * q: quotients next to representable numbers
        const double d = positive(-20, 20), q = with_exp(-20, 20);
        double x = d * q;
        for (int s = 0; s < 3; ++s, x = std::nextafter(x, x * 2)) check(x, d);
        x = fma_rn(d, q, d * q * 0x1p-53);  // ... and halfway between two
        check(x, d);
    }
    for (int t = 0; t < 1000000; ++t) {  // denominators with few or nearly all bits set
        const uint64_t m = rng() & 1 ? (1ull << (rng() % 52)) : 0xfffffffffffffull ^ (1ull << (rng() % 52));
        check(with_exp(-5, 5), real((1023ull << 52) | (m & 0xfffffffffffffull)));
    }
    const double special[] = {0.0, -0.0, 1.0, -1.0, DBL_MIN, -DBL_MIN, 5e-324, DBL_MAX, -DBL_MAX, INFINITY, -INFINITY, (double)NAN,
                              0x1p-120, 0x1p120, 0x1p-121, 0x1.fffffffffffffp119, 0x1.fffffffffffffp0, 0x1p600, 0x1p-600, 0x1p-900};
    for (double x : special)
        for (double d : special) check(x, d);
    // what plain_divisor must refuse
    for (double d : {0.0, -1.0, 0x1p120, 0x1p-121, 0x1.fffffffffffffp0, (double)NAN, (double)INFINITY})
        if (plain_divisor(d)) ++bad;
    std::printf("{\"bad\": %lld, \"fast\": %lld}\n", bad, used);
    return bad || used < 8000000 ? 1 : 0;
}
