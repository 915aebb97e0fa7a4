// lare_div.cuh -- correctly rounded division without branches, for several
// numerators over one denominator.
//
// The remap and the predictor divide several numerators by the same volume or
// density.  The forms here share the reciprocal, are straight-line and give
// the same bits:
//   rcp_fast   r = RN(1/d): three Newton-Raphson steps r + r*(1 - d*r), each
//              with the two FMAs of the cited chapters, from a seed with
//              relative error e.  A step squares the error and rounds, so two
//              of them leave e^4 and half an ulp: within one ulp for e up to
//              2^-14 (e^4 = 2^-56 is an eighth of an ulp at most).  The PTX
//              manual gives the seed 20 bits.  The third step, from an r within
//              one ulp, rounds correctly unless d's significand is all ones
//              (Markstein).
//   quot       q = RN(x/d) from r = RN(1/d) by Markstein's theorem (P.
//              Markstein, "Computation of elementary functions on the IBM
//              RISC System/6000 processor", 1990; Muller et al., "Handbook of
//              Floating-Point Arithmetic", the chapter on division by
//              Newton-Raphson iteration with an FMA): if q is a faithful
//              rounding of x/d and rem = x - d*q is formed exactly by an FMA,
//              then RN(q + rem*r) = RN(x/d).  q = RN(x*r + RN(x*e)) with
//              e = RN(r * (1 - d*r)), the part of 1/d that r misses, is within
//              half an ulp and 2^-50 of one.
// Conditions: d usable (usable_divisor: positive, exponent in -240..239, not
// all ones), and |x/d| in 2^-600..2^600 (quot_in_range on the result) or x
// zero.  Then x lies in 2^-840..2^840, x*e is zero or above 2^-710 and rem a
// multiple of 2^-944, so each is normal or exactly zero.  The callers check
// them and go back to the IEEE division otherwise, NaN and infinities included.
// (The range of d holds cells from 10^-24 to 10^24 units wide.  At exponents
// -120..119 it ended at 10^12: a 96^3 step with wider cells took 1359 us
// (resistive) and 1291 us (ideal), every op run twice, against 1308 and 1168
// with IEEE divisions only; now 910 and 784.)
#pragma once

#include <cmath>
#include <cstring>

namespace sams {
namespace dev {

// (host forms for the checks that run without a GPU)
__host__ __device__ __forceinline__ double fma_rn(double a, double b, double c)
{
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
__host__ __device__ __forceinline__ unsigned high_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x);
#else
    unsigned long long u;
    std::memcpy(&u, &x, sizeof u);
    return (unsigned)(u >> 32);
#endif
}
__host__ __device__ __forceinline__ unsigned low_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(x);
#else
    unsigned long long u;
    std::memcpy(&u, &x, sizeof u);
    return (unsigned)u;
#endif
}
// 1/d to about 20 bits (the PTX manual's figure for rcp.approx.ftz.f64, whose
// result has a zero low word).
__host__ __device__ __forceinline__ double rcp_seed(double d)
{
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    return r;
#else
    const double r = 1.0 / d;
    unsigned long long u;
    std::memcpy(&u, &r, sizeof u);
    u &= 0xffffffff00000000ull;
    double s;
    std::memcpy(&s, &u, sizeof s);
    return s;
#endif
}

// Positive, exponent in -E..E-1, not all ones.
template <unsigned E>
__host__ __device__ __forceinline__ bool divisor_within(double d)
{
    const unsigned h = high_word(d);
    return h - ((1023u - E) << 20) < ((2 * E) << 20) && !(low_word(d) == 0xffffffffu && (h & 0xfffffu) == 0xfffffu);
}
__host__ __device__ __forceinline__ bool usable_divisor(double d) { return divisor_within<240>(d); }
// (the middle of that range, from which the check of the quotients draws)
__host__ __device__ __forceinline__ bool plain_divisor(double d) { return divisor_within<120>(d); }
__host__ __device__ __forceinline__ bool quot_in_range(double q)
{
    return (high_word(q) & 0x7fffffffu) - ((unsigned)(1023 - 600) << 20) < (1200u << 20);
}
// ((h << 1) | l drops the sign)
__host__ __device__ __forceinline__ bool is_zero(double x) { return ((high_word(x) << 1) | low_word(x)) == 0; }

struct Rcp {
    double d, r, e;
};

// 1/d from the approximation r, its error squared.
__host__ __device__ __forceinline__ double newton(double d, double r) { return fma_rn(r, fma_rn(-d, r, 1.0), r); }
// RN(1/d) from a seed within 2^-14 of it.
__host__ __device__ __forceinline__ double rcp_from(double d, double seed) { return newton(d, newton(d, newton(d, seed))); }
__host__ __device__ __forceinline__ double rcp_fast(double d) { return rcp_from(d, rcp_seed(d)); }
__host__ __device__ __forceinline__ Rcp rcp_with(double d, double r)
{
    Rcp R;
    R.d = d;
    R.r = r;
    R.e = r * fma_rn(-d, r, 1.0);
    return R;
}
__host__ __device__ __forceinline__ Rcp rcp_of(double d) { return rcp_with(d, rcp_fast(d)); }

__host__ __device__ __forceinline__ double quot(double x, const Rcp &R)
{
    const double q = fma_rn(x, R.r, x * R.e);
    return fma_rn(fma_rn(-R.d, q, x), R.r, q);
}

// x / R.d with a zero numerator's sign kept (R.d positive); bad is set where
// the result may not be the IEEE quotient.
__host__ __device__ __forceinline__ double quot_check(double x, const Rcp &R, bool &bad)
{
    const double q = quot(x, R);
    const bool zero = is_zero(x);
    bad = bad || (!quot_in_range(q) && !zero);
    return zero ? x : q;
}

}  // namespace dev
}  // namespace sams
