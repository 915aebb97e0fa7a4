// lare_bc.cuh -- one (field, dimension, edge) of a built-in boundary
// condition at one ghost point, shared by the single-solve and batched fill
// kernels.
//
// The reference applies a condition to a whole edge slab as one sliced copy
// or kernel over the slab in row-major order
// (include/boundaryConditions/builtInBoundaryConditions.h: simpleClamp :55,
// simpleMirrorBC :145, simpleZeroGradientBC :224, simplePeriodicBC :252).
// Lines of the slab along the other two dimensions are independent; along the
// condition's own dimension a copy may read points the same copy writes when
// the dimension has fewer than three interior cells (e.g. a periodic upper
// edge of a half-cell field with n = 2 reads index 2 after writing it), so
// then the ghost layers of a line are filled one after another in ascending
// order, as the reference's loop does.
#pragma once

#include <string>

#include "lare_device.cuh"
#include "sams_lare_bc_other.h"

namespace sams {

// Boundary conditions of all fields as the kernels read them.  A
// SAMS_BC_LARE_OTHER slot carries its plane operations: plane pdst[q] of the
// slot's dimension receives plane psrc[q] (or zero, SAMS_PLANE_ZERO) for
// q < nplanes.
struct BcTable {
    signed char kind[SAMS_NFIELDS][3][2];
    signed char nplanes[SAMS_NFIELDS][3][2];
    int pdst[SAMS_NFIELDS][3][2][3];
    int psrc[SAMS_NFIELDS][3][2][3];
    double value[SAMS_NFIELDS][3][2];
};

// Host: set one slot of a table for a grid of n[] interior cells.  The plane
// operations of a SAMS_BC_LARE_OTHER slot must write only the edge's ghost
// planes, read planes of the field's own range, and never read a plane the
// same slot writes (so one thread per point applies them in any order).
inline bool bc_slot_set(BcTable &t, int f, int d, int e, int kind, double value, const long long n[3],
                        std::string *err)
{
    if (kind < SAMS_BC_NONE || kind > SAMS_BC_LARE_OTHER) {
        *err = "unknown boundary-condition kind";
        return false;
    }
    t.kind[f][d][e] = (signed char)kind;
    t.value[f][d][e] = value;
    t.nplanes[f][d][e] = 0;
    if (kind != SAMS_BC_LARE_OTHER) return true;
    int32_t dst[3], src[3];
    const int np = sams_lare_other_planes(f, d, e, n[d], dst, src);
    const bool half = sams_lare_field_stagger[f][d] != 0;
    const long long lb = half ? -2 : -1, ub = n[d] + 2;
    const long long glo = e == 0 ? lb : (half ? n[d] : n[d] + 1), ghi = e == 0 ? 0 : n[d] + 2;
    for (int q = 0; q < np; ++q) {
        bool ok = dst[q] >= glo && dst[q] <= ghi && (src[q] == SAMS_PLANE_ZERO || (src[q] >= lb && src[q] <= ub));
        for (int r = 0; r < np; ++r) ok = ok && src[q] != dst[r];
        if (!ok) {
            *err = "LARE BC_OTHER planes outside the field's range for this grid size";
            return false;
        }
        t.pdst[f][d][e][q] = dst[q];
        t.psrc[f][d][e][q] = src[q];
    }
    t.nplanes[f][d][e] = (signed char)np;
    return true;
}

// Host: a whole table from the C-ABI descriptor.
inline bool bc_table_from(BcTable &t, const sams_lare_bcs &bcs, const long long n[3], std::string *err)
{
    for (int f = 0; f < SAMS_NFIELDS; ++f)
        for (int d = 0; d < 3; ++d)
            for (int e = 0; e < 2; ++e)
                if (!bc_slot_set(t, f, d, e, bcs.kind[f][d][e], bcs.value[f][d][e], n, err)) return false;
    return true;
}

// Below this many interior cells in the condition's dimension an edge copy
// can read its own output: fill the ghost layers of each line in order.
constexpr int kBcSequentialBelow = 3;

struct BcEdge {
    int glo, ghi;  // ghost range of the edge in dimension d
    int dlb, dub;  // first and last domain index in dimension d
    int lo[3], hi[3];  // the slab (field range, ghost range in d)
};

__host__ __device__ inline BcEdge bc_edge_slab(const Geom &g, int f, int d, int e)
{
    const int n[3] = {g.nx, g.ny, g.nz};
    BcEdge s;
    for (int q = 0; q < 3; ++q) {
        s.lo[q] = field_half(f, q) ? -2 : -1;
        s.hi[q] = n[q] + 2;
    }
    const bool half = field_half(f, d) != 0;
    s.dlb = half ? 0 : 1;
    s.dub = n[d];
    s.glo = e == 0 ? s.lo[d] : (half ? n[d] : n[d] + 1);
    s.ghi = e == 0 ? 0 : n[d] + 2;
    s.lo[d] = s.glo;
    s.hi[d] = s.ghi;
    return s;
}

// Value the condition writes at ghost point q (q[d] in glo..ghi), from the
// array's current contents.
__host__ __device__ __forceinline__ double bc_edge_value(const double *a, const Geom &g, const BcEdge &s, int kind,
                                                double clamp_value, int d, int e, const int *q)
{
    const int gq = q[d];
    const int cnt = s.ghi - s.glo + 1;
    int p[3] = {q[0], q[1], q[2]};
    switch (kind) {
    case SAMS_BC_PERIODIC:
        p[d] = e == 0 ? s.dub - cnt + 1 + (gq - s.glo) : s.dlb + (gq - s.glo);
        return a[box_off(g, p[0], p[1], p[2])];
    case SAMS_BC_ZERO_GRADIENT:
        p[d] = e == 0 ? s.dlb : s.dub;
        return a[box_off(g, p[0], p[1], p[2])];
    case SAMS_BC_MIRROR: {
        const int last = e == 0 ? s.dlb : s.dub;
        const int first = e == 0 ? s.ghi : s.glo;
        p[d] = last;
        const double av = a[box_off(g, p[0], p[1], p[2])];
        const double bv = (av + av) / 2.0;
        p[d] = last - (gq - first);
        const double delta = a[box_off(g, p[0], p[1], p[2])] - bv;
        return bv - delta;
    }
    default:  // SAMS_BC_CLAMP
        return clamp_value;
    }
}

// Fill ghost point q, or (in a dimension with fewer than three interior
// cells) the whole ghost line through q when q is its first layer.  A LARE
// BC_OTHER slot writes q only if its plane is one the slot's operations
// write; those operations are independent, so every point is one thread.
__host__ __device__ __forceinline__ void bc_edge_apply(double *a, const Geom &g, const BcEdge &s, const BcTable &bt, int f,
                                              int d, int e, int *q)
{
    const int kind = bt.kind[f][d][e];
    const double clamp_value = bt.value[f][d][e];
    if (kind == SAMS_BC_LARE_OTHER) {
        const int np = bt.nplanes[f][d][e];
        for (int t = 0; t < np; ++t) {
            if (bt.pdst[f][d][e][t] != q[d]) continue;
            const int src = bt.psrc[f][d][e][t];
            double v = 0.0;
            if (src != SAMS_PLANE_ZERO) {
                int p[3] = {q[0], q[1], q[2]};
                p[d] = src;
                v = a[box_off(g, p[0], p[1], p[2])];
            }
            a[box_off(g, q[0], q[1], q[2])] = v;
        }
        return;
    }
    const int n = d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
    if (n >= kBcSequentialBelow) {
        const double v = bc_edge_value(a, g, s, kind, clamp_value, d, e, q);
        a[box_off(g, q[0], q[1], q[2])] = v;
        return;
    }
    if (q[d] != s.glo) return;
    for (int gq = s.glo; gq <= s.ghi; ++gq) {
        q[d] = gq;
        const double v = bc_edge_value(a, g, s, kind, clamp_value, d, e, q);
        a[box_off(g, q[0], q[1], q[2])] = v;
    }
}

// Host: whether the conditions of field f can be applied in one pass over its
// ghost shell (bc_compose_value): every ghost point's final value is then a
// function of points that the fill leaves as they are, so no thread reads
// what another writes.  That needs three or more cells in the dimension and,
// for a half-cell field, whose boundary index (0 or n) is a ghost and a
// domain point at once, conditions that leave the boundary index they read
// unchanged: both edges periodic (index 0 takes index n, which keeps its
// value), or zero-gradient, clamp or none on either.  The plane operations of
// SAMS_BC_LARE_OTHER stay with the edge by edge fill.
inline bool bc_composable(const BcTable &t, int f, const int n[3])
{
    for (int d = 0; d < 3; ++d) {
        const int l = t.kind[f][d][0], u = t.kind[f][d][1];
        if (n[d] < kBcSequentialBelow || l == SAMS_BC_LARE_OTHER || u == SAMS_BC_LARE_OTHER) return false;
        if (!field_half(f, d)) continue;
        if ((l == SAMS_BC_PERIODIC) != (u == SAMS_BC_PERIODIC) || l == SAMS_BC_MIRROR || u == SAMS_BC_MIRROR) return false;
    }
    return true;
}

// Value at point q of field f after the conditions of dimensions 0..D, lower
// edge then upper in each, from the array as it was before the fill: the last
// dimension in which q is a ghost decides, reading what the earlier
// dimensions leave at its source (the reference's order, row by row copies of
// bc_edge_value).
template <int D>
__host__ __device__ inline double bc_compose_value(const double *a, const Geom &g, const BcTable &bt, int f, int q0,
                                                   int q1, int q2)
{
    if constexpr (D < 0) {
        return a[box_off(g, q0, q1, q2)];
    } else {
        const int n = D == 0 ? g.nx : (D == 1 ? g.ny : g.nz);
        const int q = D == 0 ? q0 : (D == 1 ? q1 : q2);
        const bool half = field_half(f, D) != 0;
        auto raw = [&](int p) {
            return bc_compose_value<D - 1>(a, g, bt, f, D == 0 ? p : q0, D == 1 ? p : q1, D == 2 ? p : q2);
        };
        const int e = q >= (half ? n : n + 1) ? 1 : 0;
        if (e == 0 && q > 0) return raw(q);
        switch (bt.kind[f][D][e]) {
        case SAMS_BC_NONE:
            return raw(q);
        case SAMS_BC_PERIODIC:  // (a half-cell upper copy of index 0 reads what the lower edge put there, index n)
            return raw(e == 0 ? q + n : (half && q == n ? n : q - n));
        case SAMS_BC_ZERO_GRADIENT:
            return raw(e == 0 ? (half ? 0 : 1) : n);
        case SAMS_BC_MIRROR: {
            const double av = raw(e == 0 ? 1 : n);
            const double bv = (av + av) / 2.0;
            const double delta = raw(e == 0 ? 1 - q : 2 * n + 1 - q) - bv;
            return bv - delta;
        }
        default:  // SAMS_BC_CLAMP
            return bt.value[f][D][e];
        }
    }
}

// The points of field f's range that are ghosts in some dimension (-1 or -2
// to 0, and n+1 or, half-cell, n and up), one per t in 0 .. count-1.
struct BcShell {
    int lb[3], ext[3], nin[3], gh[3];  // first index, points, inner points 1.., ghosts per dimension
    __host__ __device__ BcShell(const Geom &g, int f)
    {
        const int n[3] = {g.nx, g.ny, g.nz};
        for (int d = 0; d < 3; ++d) {
            const int h = field_half(f, d);
            lb[d] = h ? -2 : -1;
            ext[d] = n[d] + 3 - lb[d];
            nin[d] = n[d] - h;
            gh[d] = ext[d] - nin[d];
        }
    }
    __host__ __device__ int ghost(int d, int t) const { return t < 1 - lb[d] ? lb[d] + t : nin[d] + 1 + (t - (1 - lb[d])); }
    __host__ __device__ bool point(int t, int &i, int &j, int &k) const
    {
        const int A = gh[0] * ext[1] * ext[2], B = nin[0] * gh[1] * ext[2], C = nin[0] * nin[1] * gh[2];
        if (t < A) {
            const int pl = ext[1] * ext[2], x = t / pl, r = t - x * pl;
            i = ghost(0, x);
            j = lb[1] + r / ext[2];
            k = lb[2] + r % ext[2];
            return true;
        }
        if ((t -= A) < B) {
            const int pl = gh[1] * ext[2], x = t / pl, r = t - x * pl, y = r / ext[2];
            i = 1 + x;
            j = ghost(1, y);
            k = lb[2] + (r - y * ext[2]);
            return true;
        }
        if ((t -= B) < C) {
            const int pl = nin[1] * gh[2], x = t / pl, r = t - x * pl, y = r / gh[2];
            i = 1 + x;
            j = 1 + y;
            k = ghost(2, r - y * gh[2]);
            return true;
        }
        return false;
    }
};

// The shell that the one-pass fills of several fields walk: the box -2..n+2
// outside 1..n-1 in every dimension (index n is a ghost of half-cell fields), x
// slabs, then y slabs inside x, then z slabs inside x and y.  Its points, and
// point t of it.
__host__ __device__ inline int fill_points(const Geom &g)
{
    return 6 * (g.ny + 5) * (g.nz + 5) + (g.nx - 1) * 6 * (g.nz + 5) + (g.nx - 1) * (g.ny - 1) * 6;
}
__host__ __device__ __forceinline__ int shell_index(int n, int t) { return t < 3 ? t - 2 : n + t - 3; }  // -2, -1, 0, n .. n+2
__host__ __device__ __forceinline__ bool fill_point(const Geom &g, int t, int &q0, int &q1, int &q2)
{
    const int E1 = g.ny + 5, E2 = g.nz + 5;
    const int A = 6 * E1 * E2, B = (g.nx - 1) * 6 * E2, C = (g.nx - 1) * (g.ny - 1) * 6;
    if (t < A) {
        const int x = t / (E1 * E2), r = t - x * (E1 * E2), y = r / E2;
        q0 = shell_index(g.nx, x);
        q1 = y - 2;
        q2 = r - y * E2 - 2;
        return true;
    }
    if ((t -= A) < B) {
        const int i = t / (6 * E2), r = t - i * (6 * E2), y = r / E2;
        q0 = 1 + i;
        q1 = shell_index(g.ny, y);
        q2 = r - y * E2 - 2;
        return true;
    }
    if ((t -= B) < C) {
        const int i = t / ((g.ny - 1) * 6), r = t - i * ((g.ny - 1) * 6), j = r / 6;
        q0 = 1 + i;
        q1 = 1 + j;
        q2 = shell_index(g.nz, r - j * 6);
        return true;
    }
    return false;
}

// All-periodic fields: applying the lower then upper periodic copy in x, y
// and z in turn leaves every ghost point equal to the interior point it
// wraps to, w(q) = q + n for q <= 0 and q - n for q >= n + 1 (a half-cell
// index n keeps its value), so one gather fills all ghosts of the fields in
// MASK at a point, every load issued before the first store.  (With a thread
// per field and point, the seven fills of a resistive step took 320 us at
// 256^3 and 29 us at 32^3; now 246 and 27.)
template <unsigned MASK>
__device__ __forceinline__ void periodic_copy(const Ctx &c, int q0, int q1, int q2)
{
    const Geom &g = c.g;
    const int s0 = q0 <= 0 ? q0 + g.nx : (q0 > g.nx ? q0 - g.nx : q0);
    const int s1 = q1 <= 0 ? q1 + g.ny : (q1 > g.ny ? q1 - g.ny : q1);
    const int s2 = q2 <= 0 ? q2 + g.nz : (q2 > g.nz ? q2 - g.nz : q2);
    const int dst = box_off(g, q0, q1, q2), src = box_off(g, s0, s1, s2);
    if (dst == src) return;  // (an index n: no ghost of a centred field, and kept in a half-cell one)
    const bool low0 = q0 < -1, low1 = q1 < -1, low2 = q2 < -1;  // centred dimensions start at -1
    double v[SAMS_NFIELDS];
#pragma unroll
    for (int f = 0; f < SAMS_NFIELDS; ++f)
        if ((MASK >> f) & 1u)
            if (!((low0 && !field_half(f, 0)) || (low1 && !field_half(f, 1)) || (low2 && !field_half(f, 2)))) v[f] = c.f[f][src];
#pragma unroll
    for (int f = 0; f < SAMS_NFIELDS; ++f)
        if ((MASK >> f) & 1u)
            if (!((low0 && !field_half(f, 0)) || (low1 && !field_half(f, 1)) || (low2 && !field_half(f, 2)))) c.f[f][dst] = v[f];
}

}  // namespace sams
