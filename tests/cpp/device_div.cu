// Check on the GPU of the branch-free division (lare_div.cuh, FastDiv in
// lare_device.cuh): the hardware seed is within the bound that the reciprocal
// needs, and the reciprocal, quotients, pairs and fractions have the bits of
// the IEEE operations, over random operands, quotients next to rounding
// boundaries, significands with few or nearly all bits set, and both ends of
// the ranges.  Only counters leave the kernel.
#include <cfloat>
#include <cstdint>
#include <cstdio>

#include "lare_device.cuh"

using namespace sams::dev;

struct Counts {
    unsigned long long rcp, quot, pair, frac, used, refused;
    unsigned long long seed_error;  // bits of the largest relative error of a seed
};

__device__ uint64_t mix(uint64_t z)  // splitmix64
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ double real(int exp, uint64_t significand)
{
    return __longlong_as_double((long long)(((uint64_t)(1023 + exp) << 52) | (significand & 0xfffffffffffffull)));
}

__global__ void check(long long n, uint64_t seed, Counts *out)
{
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const uint64_t a = mix(seed + 4 * (uint64_t)t), b = mix(seed + 4 * (uint64_t)t + 1), c = mix(seed + 4 * (uint64_t)t + 2),
                       e = mix(seed + 4 * (uint64_t)t + 3);
        // a divisor of -240..239, one in eight at an end of it, one in four
        // with few or nearly all bits set
        const int ed = e % 8 == 0 ? (e & 8 ? -240 : 239) : (int)((e >> 8) % 480) - 240;
        uint64_t m = a;
        if ((e >> 4) % 4 == 0) m = e & 64 ? 1ull << (a % 52) : 0xfffffffffffffull ^ (1ull << (a % 52));
        const double d = real(ed, m);
        FastDiv dv;
        const Rcp R = dv.of(d);
        if (dv.bad) {
            atomicAdd(&out->refused, 1ull);  // an all-ones significand, as good as never
            continue;
        }
        if (!same(R.r, __drcp_rn(d))) atomicAdd(&out->rcp, 1ull);
        const double err = fabs(fma_rn(-d, rcp_seed(d), 1.0));
        atomicMax(&out->seed_error, (unsigned long long)__double_as_longlong(err));
        // numerators: a quotient of -600..599, one in eight at an end, and one
        // next to a rounding boundary (d * q and its neighbours)
        const int eq = (e >> 24) % 8 == 0 ? (e & (1 << 28) ? -600 : 599) : (int)((e >> 30) % 1200) - 600;
        double x = real(eq + ed, b);
        if ((e >> 20) % 2) {
            const double q = real(eq, b);
            x = __fma_rn(d, q, (e >> 21) % 2 ? __dmul_rn(d * q, 0x1p-53) : 0.0);
            x = __longlong_as_double(__double_as_longlong(x) + (long long)(c % 5) - 2);
        }
        if (c & 8) x = -x;
        {
            FastDiv dq;
            const double q = dq(x, R), want = x / d;
            if (dq.bad ? fabs(want) > 0x1p-599 && fabs(want) < 0x1p599 : !same(q, want)) atomicAdd(&out->quot, 1ull);
            if (!dq.bad) atomicAdd(&out->used, 1ull);
        }
        {
            // a second quotient near the first in size, of either sign
            const int e2 = (int)((c >> 8) % 480) - 240, ey = eq + (int)((c >> 20) % 9) - 4;
            const double d2 = real(e2, c >> 5), y = (c & 16 ? -1.0 : 1.0) * real(ey + e2, a ^ c);
            FastDiv dp;
            const Rcp R2 = dp.of(d2);
            const double s = dp.pair(x, R, y, R2), want = x / d + y / d2;
            if (!dp.bad && !same(s, want)) atomicAdd(&out->pair, 1ull);
            if (dp.bad && usable_divisor(d2) && fabs(want) > 0x1p-599 && fabs(want) < 0x1p599) atomicAdd(&out->pair, 1ull);
        }
        {
            // a fraction of any numerator: the quotient where it is 2^-600 or
            // more (or flagged), anything below 2^-600 otherwise
            double z = real((int)((c >> 32) % 2046) - 1022, b ^ a);
            if (c % 64 == 0) z = c & 64 ? INFINITY : 0.0;
            FastDiv df;
            const double f = df.fraction(z, R), want = z / d;
            df.finite(f);
            if (!df.bad && (want >= 0x1p-600 ? !same(f, want) : !(fabs(f) <= 0x1p-599))) atomicAdd(&out->frac, 1ull);
            if (df.bad && want < 0x1p1000) atomicAdd(&out->frac, 1ull);
        }
    }
}

int main(int argc, char **)
{
    (void)argc;
    Counts h{}, *c = nullptr;
    const long long n = 32 << 20;
    bool ok = cudaMalloc(&c, sizeof h) == cudaSuccess && cudaMemset(c, 0, sizeof h) == cudaSuccess;
    if (ok) check<<<1184, 256>>>(n, 1234567, c);
    ok = ok && cudaGetLastError() == cudaSuccess && cudaMemcpy(&h, c, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess;
    double seed_error;
    static_assert(sizeof seed_error == sizeof h.seed_error, "");
    std::memcpy(&seed_error, &h.seed_error, sizeof seed_error);
    const unsigned long long bad = h.rcp + h.quot + h.pair + h.frac;
    std::printf("{\"ran\": %d, \"bad\": %llu, \"rcp\": %llu, \"quot\": %llu, \"pair\": %llu, \"frac\": %llu, \"used\": %llu, "
                "\"refused\": %llu, \"seed_error\": %.3g}\n",
                ok ? 1 : 0, bad, h.rcp, h.quot, h.pair, h.frac, h.used, h.refused, seed_error);
    return ok && bad == 0 && h.used > (unsigned long long)n * 3 / 4 && h.refused < 1000 && seed_error < 0x1p-14 ? 0 : 1;
}
