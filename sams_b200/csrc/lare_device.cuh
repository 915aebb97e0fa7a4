// lare_device.cuh -- device-side data layout and point formulas of the
// LARE3D timestep on B200.
//
// Layout: every field is one "box" over indices -2..n+2 per dimension, z
// fastest, with the z row padded so that interior index k = 1 starts on a
// 32-byte boundary (zoff = 3) and rows are a multiple of 8 doubles.  All
// fields share one geometry, so one offset serves every array.
//
// Arithmetic: this translation unit is compiled with --fmad=false and the
// formulas below keep the reference's evaluation order term by term
// (left-to-right sums, the same parenthesisation), so results are identical
// to the reference CPU build with -ffp-contract=off.  Double division and
// sqrt are IEEE round-to-nearest on the GPU as on the CPU.
#pragma once

#include <cfloat>
#include <cstdint>

#include "lare_div.cuh"
#include "sams_lare_layout.h"

namespace sams {

struct Geom {
    int nx, ny, nz;
    int sx, sy;        // element strides of i and j (k stride is 1)
    int zoff;          // k + zoff is the position of index k in its row
    long long nelem;   // doubles per field allocation
    int far;           // the solves in hand outgrow L2 (far_from_l2): fused kernels prefetch
};
// Whether arrays of this many doubles (summed over the solves stepped
// together) outgrow L2 during a phase, which reads a dozen of them.
inline int far_from_l2(long long nelem) { return nelem * 8 * 12 > 126000000LL; }

// Host/device helpers for the box geometry.
// Offsets are 32-bit: the 32 arrays of a solve must fit one GPU, so a single
// array holds far fewer than 2^31 elements (checked when a solve is set up).
__host__ __device__ inline int box_off(const Geom &g, int i, int j, int k)
{
    return (i + 2) * g.sx + (j + 2) * g.sy + (k + g.zoff);
}

// The points of a box (-2..n+2 in each dimension) outside the cube
// lo..n+hi in every dimension, one per index t in 0 .. count()-1:
// first the x slabs (whole y-z planes), then the y slabs inside the cube's
// x range, then the z slabs inside its x and y ranges.
struct BoxShell {
    int n[3];
    int lo, hi;
    __host__ __device__ long long ext(int d) const { return (long long)n[d] + 5; }
    __host__ __device__ long long in(int d) const { return (long long)n[d] + hi - lo + 1; }
    // box index of the q-th ghost layer of dimension d (lo+2 below, the rest above)
    __host__ __device__ int ghost(int d, long long q) const
    {
        return q < lo + 2 ? (int)q - 2 : n[d] + hi + 1 + (int)(q - (lo + 2));
    }
    __host__ __device__ long long count() const
    {
        return (ext(0) - in(0)) * ext(1) * ext(2) + in(0) * (ext(1) - in(1)) * ext(2) +
               in(0) * in(1) * (ext(2) - in(2));
    }
    __host__ __device__ void point(long long t, int &i, int &j, int &k) const
    {
        const long long cx = (ext(0) - in(0)) * ext(1) * ext(2);
        if (t < cx) {
            i = ghost(0, t / (ext(1) * ext(2)));
            j = (int)((t / ext(2)) % ext(1)) - 2;
            k = (int)(t % ext(2)) - 2;
            return;
        }
        t -= cx;
        const long long gy = ext(1) - in(1), cy = in(0) * gy * ext(2);
        if (t < cy) {
            i = lo + (int)(t / (gy * ext(2)));
            j = ghost(1, (t / ext(2)) % gy);
            k = (int)(t % ext(2)) - 2;
            return;
        }
        t -= cy;
        const long long gz = ext(2) - in(2);
        i = lo + (int)(t / (in(1) * gz));
        j = lo + (int)((t / gz) % in(1));
        k = ghost(2, t % gz);
    }
};

// Staggering of a field in one dimension (1 = half cell), the device-side
// copy of sams_lare_field_stagger.
__host__ __device__ constexpr int field_half(int f, int d)
{
    return (f >= SAMS_F_VX && f <= SAMS_F_VZ1) ? 1
           : (f == SAMS_F_BX) ? (d == 0)
           : (f == SAMS_F_BY) ? (d == 1)
           : (f == SAMS_F_BZ) ? (d == 2)
           : 0;
}

// 1-D axes (index i at [i + 2]); Cartesian metrics are products of these.
struct Axes {
    const double *dxb, *dyb, *dzb, *dxc, *dyc, *dzc;
};

struct Phys {
    double gamma, mu0, visc1, visc2_norm, dt_multiplier, eta_bg, eta0, j_max;
    int resistive;  // per-solve resistive flag (read by the batched launcher)
    int rke;        // remap kinetic-energy correction on (Ctx::dke allocated)
    int geometry;   // 0 Cartesian, 1 cylindrical, 2 spherical (Ctx::gf set)
    int pow2;       // Cartesian grid whose spacings are all one power of two each (Ctx::rc set)
};

// Reciprocals of the spacings and of the cell volume of a uniform Cartesian
// grid whose spacings are powers of two.  Dividing by a power of two and
// multiplying by its reciprocal give the same correctly rounded result for
// every operand, so kernels built for such grids multiply instead.
struct Recip {
    double xb, yb, zb, xc, yc, zc, cv;
    double mu0;  // 1 / mu0 (mu0 is a power of two too)
};

// Metric factors of a cylindrical or spherical solve, as LARE3D::grid builds
// them (setup.cpp:277-335), computed on the host.  All null in Cartesian
// geometry, where every factor is 1.0 and the kernels skip them.
struct GeomF {
    const double *hy, *hyc, *hyv, *xb;   // per x, index i + 2
    const double *hz, *hz1, *hz2, *hzc;  // per (x, y), index (i + 2) * (ny + 5) + (j + 2)
    const double *cot;                   // 1 / tan(yb) per y, index j + 2
};

// Per-solve device scalars.
struct Scalars {
    double dt;        // timestep of the step in progress (previous step's
                      // value until the CFL reduction has run)
    double dtr;       // LARE's dtr (equals the reduced dt)
    double dt_sub;    // resistive sub-step
    double time;      // simulation time
    unsigned long long dtmin_bits;  // running min of the CFL candidates
    long long step;
    int nsub;         // resistive sub-steps this step
    int status;       // 0 ok, nonzero: non-finite dt seen
};

// LARE uses the same 32 arrays for every solve: the 13 harness variables and
// 19 scratch arrays whose roles change with the phase of the step.
enum ScratchId {
    // Lagrangian phase
    S_CS = 0, S_RHOV, S_CSV, S_A1, S_A2, S_A3, S_VH, S_FXV, S_FYV, S_FZV,
    S_CV1, S_B1X, S_B1Y, S_B1Z, S_PE, S_PI, S_FX, S_FY, S_FZ,
    NSCRATCH
};
// Remap aliases (the whole Lagrangian scratch is dead by then).
#define S_R_CV1 S_CV1
#define S_R_CV2 S_CS
#define S_R_DB1 S_RHOV
#define S_R_RHO1 S_CSV
#define S_R_CVC1 S_A1
#define S_R_CT1 S_A2
#define S_R_CT2 S_A3
#define S_R_FE1 S_VH
#define S_R_FE2 S_FXV
#define S_R_RVN S_FYV
#define S_R_CV2N S_FZV
#define S_R_DMN S_B1X
#define S_R_V1S S_B1Y
#define S_R_FM1 S_B1Z
#define S_R_FM2 S_PE
#define S_R_FM3 S_PI

struct Ctx {
    Geom g;
    Axes ax;
    Phys p;
    double *f[13];
    double *s[NSCRATCH];
    double *dke;  // delta_ke of the rke correction (null unless Phys::rke)
    GeomF gf;     // metric factors (null in Cartesian geometry)
    Recip rc;     // reciprocals (valid when Phys::pow2)
    Scalars *sc;
};

namespace dev {

constexpr double NONE_ZERO = DBL_EPSILON;  // LARE simulationData::none_zero
constexpr double SIXTH = 1.0 / 6.0;

// An array that no thread of the running kernel writes.  Its loads take the
// read-only (non-coherent) path, so the compiler may move them across the
// kernel's stores to other arrays and keep more of them in flight.
struct RO {
    const double *p;
    __device__ __forceinline__ double operator[](int i) const { return __ldg(p + i); }
};

// How an op divides.  FastDiv: straight-line (lare_div.cuh); `bad` says that
// some quotient may not be the IEEE one, and the caller then runs the op again
// with IeeeDiv before anything it reads has been overwritten.  of() takes a
// denominator, the call divides by it; pair() is the sum of two quotients of
// non-negative numerators and fraction() x / d, x not negative, where a result below 2^-600,
// added to or taken from one or two, may be anything below that.
//
// With IEEE divisions throughout, against now (us, 256^3 power-of-two grid / 96^3):
// predictor 1451 / 154 -> 1233 / 129, x stages 1239 / 85 -> 1051 / 71, y stages
// 1367 / 93 -> 1198 / 81, z stages 1367 / 116 -> 1257 / 86, edge viscosity
// 866 / 52 -> 767 / 48, corrector 597 / 38 -> 540 / 32; k_visc_split
// (three blocks per SM) 1090 / 86 -> 1040 / 73.  (The reciprocal's third Newton
// step, added since, costs up to 2% of a kernel: predictor 1248 at 256^3.)
struct IeeeDiv {
    static constexpr bool bad = false;
    struct R {
        double d;
    };
    __host__ __device__ __forceinline__ R of(double d) { return R{d}; }
    __host__ __device__ __forceinline__ double operator()(double x, const R &r) { return x / r.d; }
    __host__ __device__ __forceinline__ double pair(double x, const R &r, double y, const R &q) { return x / r.d + y / q.d; }
    __host__ __device__ __forceinline__ double fraction(double x, const R &r) { return x / r.d; }
    __host__ __device__ __forceinline__ void finite(double) {}
};
struct FastDiv {
    bool bad = false;
    using R = Rcp;
    __host__ __device__ __forceinline__ R of(double d)
    {
        bad = bad || !usable_divisor(d);
        return rcp_of(d);
    }
    __host__ __device__ __forceinline__ double operator()(double x, const R &r) { return quot_check(x, r, bad); }
    __host__ __device__ __forceinline__ double pair(double x, const R &r, double y, const R &q)
    {
        const double s = quot(x, r) + quot(y, q);
        const bool zero = ((high_word(x) << 1) | low_word(x) | (high_word(y) << 1) | low_word(y)) == 0;
        bad = bad || (!quot_in_range(s) && !zero);
        return s;
    }
    __host__ __device__ __forceinline__ double fraction(double x, const R &r) { return quot(x, r); }
    // (an infinity or NaN out of fraction() is left to the IEEE run)
    __host__ __device__ __forceinline__ void finite(double q) { bad = bad || (high_word(q) & 0x7fffffffu) >= 0x7ff00000u; }
};

// A denominator made of spacings: on power-of-two grids (P2) the product with
// its exact reciprocal r (Recip), elsewhere the division.
template <bool P2, class DV>
struct By {
    typename DV::R R;
    double r;
    __device__ __forceinline__ By(DV &dv, double d, double r_)
    {
        if constexpr (!P2) R = dv.of(d);
        r = r_;
    }
    __device__ __forceinline__ double operator()(DV &dv, double x) const
    {
        if constexpr (P2) return x * r;
        else return dv(x, R);
    }
};

// portableWrapper min/max semantics (include/pp/utils.h:277-335).
__device__ __forceinline__ double pmin(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double pmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double pmin_list3(double a, double b, double c)
{
    double m = a;
    if (b < m) m = b;
    if (c < m) m = c;
    return m;
}
__device__ __forceinline__ double pmin_list4(double a, double b, double c, double d)
{
    double m = a;
    if (b < m) m = b;
    if (c < m) m = c;
    if (d < m) m = d;
    return m;
}

// The upwind one of two values as the reference picks it, a * vad_p + b * vad_m
// with weights one and zero: the chosen value plus zero times the other, one
// fused multiply-add whose product is exact, so signed zeros, infinities and
// NaN come out as they do there.
__device__ __forceinline__ double pick(bool up, double a, double b) { return fma_rn(up ? b : a, 0.0, up ? a : b); }

// One face along a sweep as its upwind fluxes see it: up where the flow goes
// up the sweep, phi the swept fraction, ci the cell length at the face and cu
// the upwind one, bu the upwind volume.
template <class DV>
struct Face {
    bool up;
    double phi;
    typename DV::R ci, cu;
    double bu;
};

// The van Leer limited correction Di of every remap flux function (e.g.
// xremap.cpp:305-316) and the upwind value fu.
template <class DV>
__device__ __forceinline__ double limited(DV &dv, const Face<DV> &F, double fm, double fi, double fp, double fp2,
                                          double &fu)
{
    const double dfm = fi - fm, dfi = fp - fi, dfp = fp2 - fp;
    fu = pick(F.up, fi, fp);
    const double dfu = pick(F.up, dfm, dfp);
    const double Da = dv.pair((2.0 - F.phi) * fabs(dfi), F.ci, (1.0 + F.phi) * fabs(dfu), F.cu) * SIXTH;
    // sign_v * ss * min, with ss = 0.5 * (sign(dfi) + sign(dfu)): the minimum
    // with the product's sign, or a zero with sign_v's where the slopes differ
    const double m = pmin_list3(fabs(Da) * F.bu, fabs(dfi), fabs(dfu));
    const bool pi = dfi >= 0.0, pu = dfu >= 0.0;
    const double v = F.up ? 1.0 : -1.0;
    return (pi == pu ? (pi ? v : -v) : 0.0 * v) * m;
}

// Evans-Hawley constrained-transport flux of a transverse face field
// (vx_by_flux xremap.cpp:269-319 and the five analogues in x/y/zremap.cpp),
// from the four quotients b/db along the sweep, and the mass flux through a
// face (x_mass_flux xremap.cpp:373-422 and analogues): o_v is the swept
// length or volume.
template <class DV>
__device__ __forceinline__ double swept_flux(DV &dv, const Face<DV> &F, double o_v, double fm, double fi, double fp,
                                             double fp2)
{
    double fu;
    const double Di = limited(dv, F, fm, fi, fp, fp2, fu);
    return (fu + Di * (1.0 - F.phi)) * o_v;
}

// Specific-energy flux (x_energy_flux xremap.cpp:429-483 and analogues) and
// momentum flux (x_mom_flux xremap.cpp:485-566 and analogues) before their
// product with dm; dmu is the swept mass fraction.
template <class DV>
__device__ __forceinline__ double carried(DV &dv, const Face<DV> &F, double fm, double fi, double fp, double fp2, double dmu)
{
    double fu;
    const double Di = limited(dv, F, fm, fi, fp, fp2, fu);
    return fu + Di * (1.0 - dmu);
}

// |dm| / dxbu / rhou (the z sweep's momentum flux divides by dxbu * rhou in
// one step, zremap.cpp:509).
template <bool ZFORM, class DV>
__device__ __forceinline__ double mass_fraction(DV &dv, double dm, const typename DV::R &bu, double rhou)
{
    double dmu;
    if constexpr (ZFORM) dmu = dv.fraction(fabs(dm), dv.of(bu.d * rhou));
    else dmu = dv.fraction(dv.fraction(fabs(dm), bu), dv.of(rhou));
    dv.finite(dmu);
    return dmu;
}

// Caramana edge viscosity (lagran.cpp:56-93).  v[a] are the four points
// along the edge direction, o1/o2 the edge ends.
template <bool P2, class DV, class A>
__device__ __forceinline__ double edge_viscosity(DV &div, double dt, double visc1, double v2n, const A &vx,
                                                 const A &vy, const A &vz, const A &rho_v,
                                                 double dvdots, double dx, double dxm, double dxp,
                                                 double cs_edge, int o0, int o1, int o2, int o3, double rdx = 0.0)
{
    dvdots = pmin(0.0, dvdots);
    double rv1 = rho_v[o1], rv2 = rho_v[o2];
    double rho_edge = div(2.0 * rv1 * rv2, div.of(rv1 + rv2));
    double vx1 = vx[o1], vx2 = vx[o2], vy1 = vy[o1], vy2 = vy[o2], vz1 = vz[o1], vz2 = vz[o2];
    double dvx = vx1 - vx2, dvy = vy1 - vy2, dvz = vz1 - vz2;
    double dv2 = dvx * dvx + dvy * dvy + dvz * dvz;
    double dv = sqrt(dv2);
    bool small = (P2 ? dv * dt * rdx : div(dv * dt, div.of(dx))) < 1.e-14;
    // (where the jump is too small its quotients are not used: divide by one)
    dvdots = small ? 0.0 : div(dvdots, div.of(small ? 1.0 : dv));
    double dvxm = vx[o0] - vx1, dvxp = vx2 - vx[o3];
    double dvym = vy[o0] - vy1, dvyp = vy2 - vy[o3];
    double dvzm = vz[o0] - vz1, dvzp = vz2 - vz[o3];
    double rl = div((dvxp * dvx + dvyp * dvy + dvzp * dvz) * dx, div.of(small ? 1.0 : dxp * dv2));
    double rr = div((dvxm * dvx + dvym * dvy + dvzm * dvz) * dx, div.of(small ? 1.0 : dxm * dv2));
    if (small) rl = rr = 1.0;
    double psi = pmin_list4(0.5 * (rr + rl), 2.0 * rl, 2.0 * rr, 1.0);
    psi = pmax(0.0, psi);
    double q_k_bar = rho_edge * (v2n * dv + sqrt(v2n * v2n * dv2 + (visc1 * cs_edge) * (visc1 * cs_edge)));
    return q_k_bar * (1.0 - psi) * dvdots;
}

}  // namespace dev
}  // namespace sams
