// Host check of FastDiv (lare_device.cuh) over the scales it takes: divisors of
// exponents -240..239 and quotients in 2^-600..2^600 stay on the straight path
// and give the IEEE bits; what lies outside is flagged.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "lare_device.cuh"

using namespace sams::dev;

static long long bad = 0;
static uint64_t bits(double x)
{
    uint64_t u;
    std::memcpy(&u, &x, sizeof u);
    return u;
}

int main()
{
    std::mt19937_64 rng(17);
    auto real = [&](int exp) {  // a random significand
        const uint64_t u = ((uint64_t)(1023 + exp) << 52) | (rng() & 0xfffffffffffffull);
        double x;
        std::memcpy(&x, &u, sizeof x);
        return x;
    };
    auto between = [&](int lo, int hi) { return lo + (int)(rng() % (uint64_t)(hi - lo + 1)); };
    auto sign = [&](double x) { return rng() & 1 ? -x : x; };
    for (int t = 0; t < 3000000; ++t) {
        const int ed = t % 4 == 0 ? (t % 8 ? -240 : 239) : between(-240, 239);
        const int eq = t % 5 == 0 ? (t % 10 ? -599 : 598) : between(-599, 598);
        const double d = real(ed), x = sign(real(eq + ed));
        FastDiv dv;
        const FastDiv::R R = dv.of(d);
        const double q = dv(x, R);
        if (dv.bad || bits(q) != bits(x / d)) ++bad;
        // two quotients of one scale, the second numerator of either sign
        const double d2 = real(between(-240, 239)), y = sign(std::fabs(q) * d2 * real(between(-3, 3)));
        if (std::isfinite(y) && std::fabs(y / d2) > 0x1p-590 && std::fabs(y / d2) < 0x1p590) {
            FastDiv dp;
            const double s = dp.pair(x, R, y, dp.of(d2)), want = x / d + y / d2;
            if (!dp.bad && bits(s) != bits(want)) ++bad;
            if (dp.bad && std::fabs(want) > 0x1p-599 && std::fabs(want) < 0x1p599) ++bad;
        }
        // a fraction of any size: the quotient, or below 2^-600 anything there
        const double f = dv.fraction(std::fabs(x), R), z = real(between(-1022, 1023));
        if (bits(f) != bits(std::fabs(x) / d)) ++bad;
        FastDiv df;
        const double g = df.fraction(z, R), wz = z / d;
        df.finite(g);
        if (wz >= 0x1p-600 ? !df.bad && bits(g) != bits(wz) : !(std::fabs(g) <= 0x1p-599)) ++bad;
        if (!df.bad && !std::isfinite(wz)) ++bad;
    }
    // outside the range of divisors and quotients
    for (double d : {0.0, -1.0, 0x1p240, 0x1.fffffffffffffp-241, 0x1.fffffffffffffp3, (double)NAN, (double)INFINITY}) {
        FastDiv dv;
        dv.of(d);
        if (!dv.bad) ++bad;
    }
    for (double x : {0x1p601, 0x1p-601, DBL_MIN, 5e-324, (double)NAN, (double)INFINITY}) {
        FastDiv dv;
        dv(x, dv.of(1.0));
        if (!dv.bad) ++bad;
    }
    // the ends, and zeros of both signs
    for (double d : {0x1p-240, 0x1.ffffffffffffep239})
        for (double x : {0.0, -0.0, 0x1p-599, 0x1p599}) {
            FastDiv dv;
            const double q = dv(x * d, dv.of(d));
            if (dv.bad || bits(q) != bits(x * d / d)) ++bad;
        }
    std::printf("{\"bad\": %lld}\n", bad);
    return bad ? 1 : 0;
}
