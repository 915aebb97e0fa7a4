// lare_solver.cu -- kernels and step orchestration of one LARE3D solve.
//
// One step on the device, in launch order (reference events in brackets;
// bodies of the fused kernels in lare_march.cuh):
//   [startOfTimestep -> lagrangian_step, lagran.cpp:95-173]
//     k_cellnode_march (CellPrep + NodePrep), Alpha, k_visc_split (Visc +
//     CFL block minima), k_dt_finalize, resistive only: 2 x {k_resist_march
//     (ResistRK + ResistB), fill B + energies}, k_pred_march (Pred1 + Pred2),
//     fill v1
//   [halfTimestep -> corrector_step, lagran.cpp:739-804]
//     k_heat_march (Corr1 from per-node edge terms), Corr2, fill v +
//     energies + rho
//   [endOfTimestep -> eulerian_remap, remap.cpp:23-111]
//     x: k_cellnode_march (SweepVol + SweepCvc), k_ctmass (CT and mass
//        fluxes, dm's ghosts along x), k_psweep (S6-S8 out of place, with
//        SweepCTUpd bringing B to flux form), fill the nine state fields
//     y: the same along y
//     z: k_cellnode_march, k_ctmass_z, k_zsweep (S6-S8 in place, with
//        SweepCTUpd bringing B back from flux form), fill
// A fill is one launch (k_bc_periodic, k_bc_compose) unless conditions do not
// compose (k_bc_edge, one launch per dimension and edge).  With rke the
// sweeps' stages are separate kernels (SweepS6/S7/S8, the rke kernels); with
// a B edge that has no condition, or fewer than three cells somewhere, B is
// scaled by passes of its own (BScale) and k_copy_shell completes the
// out-of-place arrays.
// The runner's step++/time += dt (runner.h:573-574) happens in k_dt_finalize.
// Nothing is read back to the host inside a step.
#include "lare_solver.cuh"
#include "lare_ops.cuh"
#include "lare_march.cuh"
#include "lare_bc.cuh"
#include "lare_geom_host.h"
#include "lare_repack.cuh"

#include <algorithm>
#include <cstdio>
#include <cstring>

namespace sams {

namespace {

constexpr int kThreads = 256;

// One thread per (j, k) of a plane, blockIdx.y walks i.  GEO: the solve's
// geometry is curvilinear (its metric factors are applied); the Cartesian
// instantiation has no trace of them.
template <class Op, bool GEO, bool P2>
__global__ void __launch_bounds__(kThreads, Op::kMinBlocks) k_op(const __grid_constant__ Ctx c, int arg)
{
    int lo[3], hi[3];
    Op::bounds(c.g, arg, lo, hi);
    const int nk = hi[2] - lo[2] + 1;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long plane = (long long)(hi[1] - lo[1] + 1) * nk;
    if (t >= plane) return;
    const int j = lo[1] + (int)(t / nk);
    const int k = lo[2] + (int)(t % nk);
    for (int i = lo[0] + (int)blockIdx.y; i <= hi[0]; i += gridDim.y) Op::template run<GEO, P2>(c, arg, i, j, k);
}

// The fused kernels (bodies in lare_march.cuh), one block of the phase per
// CUDA block.
using march::kMThreads;
using march::kRP;
using march::kZThreads;
using march::MarchTile;
using march::PrepMarch;
using march::VolMarch;
using march::WinTile;
using march::ZTile;

template <bool GEO, bool P2, int CW>
__global__ void __launch_bounds__(kMThreads, 3) k_pred_march(const __grid_constant__ Ctx c, MarchTile m, int resistive, double *pe_out, double *pi_out)
{
    extern __shared__ double ring[];
    march::pred<GEO, P2, CW>(c, m, (int)blockIdx.x, resistive, pe_out, pi_out, ring);
}

template <class P, bool GEO, bool P2, int CW>
__global__ void __launch_bounds__(kMThreads, P::kMinBlocks) k_cellnode_march(const __grid_constant__ Ctx c, MarchTile m, int arg)
{
    extern __shared__ double ring[];
    march::cellnode<P, GEO, P2, CW>(c, m, (int)blockIdx.x, arg, ring);
}

template <bool GEO, bool P2, int CW>
__global__ void __launch_bounds__(kMThreads, march::kHeatMinBlocks) k_heat_march(const __grid_constant__ Ctx c, MarchTile m)
{
    extern __shared__ double ring[];
    march::heat_edges<GEO, P2, CW>(c, m, (int)blockIdx.x, ring);
}

template <bool GEO, bool P2, int CW>
__global__ void __launch_bounds__(kMThreads, P2 ? 5 : 4) k_resist_march(const __grid_constant__ Ctx c, MarchTile m, double *nbx, double *nby, double *nbz)
{
    extern __shared__ double ring[];
    march::resist<GEO, P2, CW>(c, m, (int)blockIdx.x, nbx, nby, nbz, ring);
}

template <int DIR, bool GEO>
__global__ void __launch_bounds__(ops::kWinThreads, 5) k_ctmass(const __grid_constant__ Ctx c, WinTile w, int scale, int images)  // cap tuned on B200
{
    extern __shared__ double csm[];
    march::ctmass<DIR, GEO>(c, w, (int)blockIdx.x, scale, images, csm);
}

template <bool GEO>
__global__ void __launch_bounds__(march::kZCtThreads, 4) k_ctmass_z(const __grid_constant__ Ctx c, ZTile z, int images)
{
    __shared__ double zsm[ops::SweepCTMass<2>::NARR * march::kZCtThreads];
    march::ctmass_z<GEO>(c, z, (int)blockIdx.x, images, zsm);
}

template <int DIR, bool GEO>
__global__ void __launch_bounds__(ops::kWinThreads, 4) k_psweep(const __grid_constant__ Ctx c, WinTile wt, ops::SweepOut w, int ct_arg)  // window shape and cap tuned on B200
{
    extern __shared__ double psm[];
    march::psweep<DIR, GEO>(c, wt, (int)blockIdx.x, w, ct_arg, psm);
}

template <bool GEO>
__global__ void __launch_bounds__(kZThreads, 4) k_zsweep(const __grid_constant__ Ctx c, int ct_arg)  // 4 blocks per SM: 96^3 133 -> 116 us, 256^3 1.45 -> 1.36 ms against 5; 3 was 10% slower
{
    extern __shared__ double zsm[];
    march::zsweep<GEO>(c, (int)blockIdx.x, ct_arg, zsm);
}

// The points of the out-of-place sweep's arrays it does not compute (rho and
// energies outside 1..n, velocities outside 0..n in some dimension): copied
// from the solve's arrays, so the new arrays are complete boxes.  One
// thread per shell point: the rho / energy shell, then the velocity shell.
__global__ void __launch_bounds__(kThreads) k_copy_shell(const __grid_constant__ Ctx c, ops::SweepOut w)
{
    ops::copy_shell(c, c.g, w, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

// Visc with two threads per cell: a block holds 128 consecutive (j, k)
// points of a y-z plane (walking i); its first four warps run the viscous heating and forces
// (ops::Visc::heat_forces), the other four the viscous pressure and CFL
// candidate (ops::Visc::cfl), so each thread carries half the work's live
// values.  Both halves read the same corners, which the block's L1 serves.
// The block's minimum candidate goes to Scalars::dtmin_bits: positive
// doubles order like their bit patterns, so an integer atomicMin is an
// exact, order-free minimum.
template <bool GEO, bool P2>
__global__ void __launch_bounds__(kThreads, 3) k_visc_split(const __grid_constant__ Ctx c)
{
    int lo[3], hi[3];
    ops::Visc::bounds(c.g, 0, lo, hi);
    const int nk = hi[2] - lo[2] + 1;
    const int half = (int)threadIdx.x >> 7;
    const long long t = (long long)blockIdx.x * (kThreads / 2) + (threadIdx.x & (kThreads / 2 - 1));
    const long long plane = (long long)(hi[1] - lo[1] + 1) * nk;
    double best = DBL_MAX;
    bool bad = false;
    if (t < plane) {
        const int j = lo[1] + (int)(t / nk);
        const int k = lo[2] + (int)(t % nk);
        for (int i = lo[0] + (int)blockIdx.y; i <= hi[0]; i += gridDim.y) {
            if (c.g.far && i + (int)gridDim.y <= hi[0]) {  // the plane this thread walks to next
                const int o = box_off(c.g, i + (int)gridDim.y, j, k);
                if (half == 0) {
                    march::prefetch(c.f[SAMS_F_VX], o);
                    march::prefetch(c.f[SAMS_F_VY], o);
                    march::prefetch(c.f[SAMS_F_VZ], o);
                    march::prefetch(c.s[S_A1], o);
                    march::prefetch(c.s[S_A2], o);
                    march::prefetch(c.s[S_A3], o);
                } else {
                    march::prefetch(c.f[SAMS_F_BX], o);
                    march::prefetch(c.f[SAMS_F_BY], o);
                    march::prefetch(c.f[SAMS_F_BZ], o);
                    march::prefetch(c.f[SAMS_F_RHO], o);
                    march::prefetch(c.f[SAMS_F_ENERGY_ELECTRON], o);
                    march::prefetch(c.f[SAMS_F_ENERGY_ION], o);
                }
            }
            if (half == 0)
                ops::Visc::heat_forces<GEO, P2>(c, i, j, k, bad);
            else if (i <= c.g.nx && j <= c.g.ny && k <= c.g.nz)
                best = dev::pmin(best, ops::Visc::cfl<GEO, P2>(c, i, j, k, bad));
        }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&c.sc->status, 1);
    for (int off = 16; off > 0; off >>= 1) best = dev::pmin(best, __shfl_xor_sync(0xffffffffu, best, off));
    __shared__ double wmin[kThreads / 32];
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = wmin[0];
        for (int w = 1; w < kThreads / 32; ++w) m = dev::pmin(m, wmin[w]);
        if (m < DBL_MAX) atomicMin(&c.sc->dtmin_bits, (unsigned long long)__double_as_longlong(m));
    }
}

// dt = dt_multiplier * min (lagran.cpp:387-442), then the runner's
// min-with-DBL_MAX (runner.h:161-167, shared_data.h:428-440); the resistive
// sub-step is dt / (int(dt/dtr) + 1) (lagran.cpp:159-163); dtr == dt, so
// that count is 2.  Also the runner's time += dt, step++.
__global__ void k_dt_finalize(Scalars *sc, double dt_multiplier, int resistive)
{
    double m = __longlong_as_double((long long)sc->dtmin_bits);
    double dt = dt_multiplier * m;
    sc->dtr = dt;
    dt = dt < DBL_MAX ? dt : DBL_MAX;
    sc->dt = dt;
    if (resistive) {
        int nsub = (int)(dt / sc->dtr) + 1;
        sc->nsub = nsub;
        sc->dt_sub = dt / (double)nsub;
    }
    sc->dtmin_bits = (unsigned long long)__double_as_longlong(DBL_MAX);
    if (!(m < DBL_MAX) || !(dt > 0.0) || !(dt < DBL_MAX)) sc->status = 1;
    sc->time += dt;
    sc->step += 1;
}

// ---------------------------------------------------------------------------
// Boundary fills (variableDef::applyBoundaryConditions order,
// include/harness/variableDef.h:539-605; built-in conditions of
// include/boundaryConditions/builtInBoundaryConditions.h).
// ---------------------------------------------------------------------------

struct FieldList {
    int n;
    int id[SAMS_NFIELDS];
};

// All-periodic fields, one thread per point of the shell (periodic_copy).
template <unsigned MASK>
__global__ void __launch_bounds__(kThreads) k_bc_periodic(const __grid_constant__ Ctx c)
{
    int q0, q1, q2;
    if (fill_point(c.g, (int)(blockIdx.x * blockDim.x + threadIdx.x), q0, q1, q2)) periodic_copy<MASK>(c, q0, q1, q2);
}

// One (dimension, edge) of the given fields, exactly as the reference's
// boundary-condition objects apply it (lare_bc.cuh).
__global__ void __launch_bounds__(kThreads) k_bc_edge(const __grid_constant__ Ctx c, FieldList fl, BcTable bt, int d, int e)
{
    const int f = fl.id[blockIdx.y];
    const int kind = bt.kind[f][d][e];
    if (kind == SAMS_BC_NONE) return;
    const Geom &g = c.g;
    const BcEdge sl = bc_edge_slab(g, f, d, e);
    const int e1 = sl.hi[1] - sl.lo[1] + 1, e2 = sl.hi[2] - sl.lo[2] + 1;
    const long long total = (long long)(sl.hi[0] - sl.lo[0] + 1) * e1 * e2;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    int q[3];
    q[0] = sl.lo[0] + (int)(t / ((long long)e1 * e2));
    q[1] = sl.lo[1] + (int)((t / e2) % e1);
    q[2] = sl.lo[2] + (int)(t % e2);
    bc_edge_apply(c.f[f], g, sl, bt, f, d, e, q);
}

// All conditions of the given fields in one pass over each field's ghost
// shell, where they compose (bc_composable): the six edge launches of a fill
// with walls become one.
__global__ void __launch_bounds__(kThreads) k_bc_compose(const __grid_constant__ Ctx c, FieldList fl, BcTable bt)
{
    const int f = fl.id[blockIdx.y];
    const BcShell sh(c.g, f);
    int i, j, k;
    if (!sh.point((int)(blockIdx.x * blockDim.x + threadIdx.x), i, j, k)) return;
    double *a = c.f[f];
    const double v = bc_compose_value<2>(a, c.g, bt, f, i, j, k);
    a[box_off(c.g, i, j, k)] = v;
}

FieldList make_list(unsigned mask)
{
    FieldList fl{};
    for (int f = 0; f < SAMS_NFIELDS; ++f)
        if (mask & (1u << f)) fl.id[fl.n++] = f;
    return fl;
}

long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

// Whether n values split into tiles of w lanes keep at least three quarters
// of the lanes busy.
bool lanes_full(long long n, long long w) { return 4 * n >= 3 * w * ceil_div(n, w); }

}  // namespace

// ---------------------------------------------------------------------------

long long Solver::bytes_for(const sams_lare_params &p)
{
    const long long zrow = ((p.nz + 6) + 7) / 8 * 8;
    const long long nelem = (p.nx + 5) * (p.ny + 5) * zrow;
    const long long narr = SAMS_NFIELDS + NSCRATCH + (p.rke ? 1 : 0);
    const long long staging = (p.nx + 5) * (p.ny + 5) * (p.nz + 5);
    long long axes = 6 * (p.nx + p.ny + p.nz + 18);
    if (p.geometry) axes += 5 * (p.nx + 6) * (p.ny + 6) + 8 * (p.nx + p.ny + 12);
    return (narr * nelem + staging + axes) * (long long)sizeof(double) + (long long)sizeof(Scalars) + 4096;
}

bool Solver::own_stream(const sams_lare_params &p) { return lanes_full(p.nz + 1, 31); }

Solver::~Solver() { free_all(); }

void Solver::free_all()
{
    if (device_ >= 0) cudaSetDevice(device_);
    for (auto &kv : graphs_) cudaGraphExecDestroy(kv.second);
    graphs_.clear();
    if (arena_) cudaFree(arena_);
    if (axes_) cudaFree(axes_);
    if (sc_) cudaFree(sc_);
    if (staging_) cudaFree(staging_);
    if (own_stream_) cudaStreamDestroy(own_stream_);
    arena_ = nullptr;
    axes_ = nullptr;
    sc_ = nullptr;
    staging_ = nullptr;
    own_stream_ = nullptr;
}

int Solver::check(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return SAMS_OK;
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? SAMS_ERR_NOMEM : SAMS_ERR_CUDA;
}

static void axis_host(double lo, double hi, long long n, std::vector<double> &db, std::vector<double> &dc)
{
    // axisRegistry: b(i) = lo + d*i, c(i) = 0.5*(b(i) + b(i-1)), deltas with
    // the first one copied from the next (non-periodic axes).
    std::vector<double> b(n + 5), c(n + 5);
    double d = (hi - lo) / (double)n;
    for (long long i = -2; i <= n + 2; ++i) b[i + 2] = lo + d * (double)i;
    for (long long i = -1; i <= n + 2; ++i) c[i + 2] = 0.5 * (b[i + 2] + b[i + 1]);
    db.assign(n + 6, 0.0);
    dc.assign(n + 6, 0.0);
    for (long long i = -1; i <= n + 2; ++i) db[i + 2] = b[i + 2] - b[i + 1];
    db[0] = db[1];
    for (long long i = 0; i <= n + 2; ++i) dc[i + 2] = c[i + 2] - c[i + 1];
    dc[1] = dc[2];
}

int Solver::init(const sams_lare_params &p, const sams_lare_bcs &bcs, int device)
{
    return init_impl(p, bcs, device, nullptr);
}

int Solver::init_slab(const sams_lare_params &p, const sams_lare_bcs &bcs, int device, const XSlab &slab)
{
    if (slab.off < 0 || slab.off + p.nx > slab.nx_global) {
        err = "slab outside the grid";
        return SAMS_ERR_INVALID;
    }
    if (p.rke) {
        err = "the remap kinetic-energy correction (rke) gathers over the whole grid in order; not on slabs";
        return SAMS_ERR_UNSUPPORTED;
    }
    return init_impl(p, bcs, device, &slab);
}

int Solver::init_impl(const sams_lare_params &p, const sams_lare_bcs &bcs, int device, const XSlab *slab)
{
    if (p.nx < 1 || p.ny < 1 || p.nz < 1) { err = "grid sizes must be >= 1"; return SAMS_ERR_INVALID; }
    if (p.nx > 60000 || p.ny > 60000 || p.nz > 60000) { err = "grid size too large"; return SAMS_ERR_INVALID; }
    if (p.geometry < 0 || p.geometry > 2) { err = "geometry must be 0 (Cartesian), 1 (cylindrical) or 2 (spherical)"; return SAMS_ERR_UNSUPPORTED; }
    if (!(p.x_max > p.x_min) || !(p.y_max > p.y_min) || !(p.z_max > p.z_min)) {
        err = "empty domain";
        return SAMS_ERR_INVALID;
    }
    p_ = p;
    device_ = device;
    {
        const long long n[3] = {p.nx, p.ny, p.nz};
        if (!bc_table_from(bc_, bcs, n, &err)) return SAMS_ERR_INVALID;
    }
    int rc;
    if ((rc = check(cudaSetDevice(device), "cudaSetDevice"))) return rc;
    if ((rc = check(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device), "sm count")))
        return rc;
    if ((rc = check(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking), "cudaStreamCreate"))) return rc;
    stream_ = own_stream_;

    Geom &g = ctx_.g;
    g.nx = (int)p.nx;
    g.ny = (int)p.ny;
    g.nz = (int)p.nz;
    g.zoff = 3;
    const long long zrow = ((p.nz + 6) + 7) / 8 * 8;
    const long long sx = (long long)(p.ny + 5) * zrow;
    if ((long long)(p.nx + 5) * sx > INT32_MAX) {
        err = "one array of this grid exceeds 2^31 elements";
        return SAMS_ERR_UNSUPPORTED;
    }
    g.sy = (int)zrow;
    g.sx = (int)sx;
    g.nelem = (long long)(p.nx + 5) * sx;
    g.far = far_from_l2(g.nelem);
    // the rke correction keeps one more array (delta_ke) across the sweeps
    const long long narr = SAMS_NFIELDS + NSCRATCH + (p.rke ? 1 : 0);
    const size_t abytes = (size_t)narr * (size_t)g.nelem * sizeof(double);
    if ((rc = check(cudaMalloc(&arena_, abytes), "cudaMalloc(state)"))) return rc;
    if ((rc = check(cudaMemsetAsync(arena_, 0, abytes, stream_), "cudaMemset(state)"))) return rc;
    for (int f = 0; f < SAMS_NFIELDS; ++f) ctx_.f[f] = arena_ + (size_t)f * g.nelem;
    for (int s = 0; s < NSCRATCH; ++s) ctx_.s[s] = arena_ + (size_t)(SAMS_NFIELDS + s) * g.nelem;
    ctx_.dke = p.rke ? arena_ + (size_t)(SAMS_NFIELDS + NSCRATCH) * g.nelem : nullptr;

    // 1-D spacings: dxb, dyb, dzb, dxc, dyc, dzc, each (n + 6) long.
    std::vector<double> dxb, dyb, dzb, dxc, dyc, dzc;
    if (slab) {  // the whole grid's x axis from the slab's offset on
        std::vector<double> gb, gc;
        axis_host(p.x_min, p.x_max, slab->nx_global, gb, gc);
        dxb.assign(gb.begin() + slab->off, gb.begin() + slab->off + p.nx + 6);
        dxc.assign(gc.begin() + slab->off, gc.begin() + slab->off + p.nx + 6);
    } else {
        axis_host(p.x_min, p.x_max, p.nx, dxb, dxc);
    }
    axis_host(p.y_min, p.y_max, p.ny, dyb, dyc);
    axis_host(p.z_min, p.z_max, p.nz, dzb, dzc);
    std::vector<double> packed;
    for (auto *v : {&dxb, &dyb, &dzb, &dxc, &dyc, &dzc}) packed.insert(packed.end(), v->begin(), v->end());
    const size_t geo_off = packed.size();
    if (p.geometry) {  // metric factors after the spacings
        std::vector<double> t = slab ? geom_tables_slab(p, slab->off, slab->nx_global) : geom_tables(p);
        packed.insert(packed.end(), t.begin(), t.end());
    }
    if ((rc = check(cudaMalloc(&axes_, packed.size() * sizeof(double)), "cudaMalloc(axes)"))) return rc;
    if ((rc = check(cudaMemcpy(axes_, packed.data(), packed.size() * sizeof(double), cudaMemcpyHostToDevice), "axes upload"))) return rc;
    size_t off = 0;
    const double **slots[6] = {&ctx_.ax.dxb, &ctx_.ax.dyb, &ctx_.ax.dzb, &ctx_.ax.dxc, &ctx_.ax.dyc, &ctx_.ax.dzc};
    const size_t lens[6] = {dxb.size(), dyb.size(), dzb.size(), dxc.size(), dyc.size(), dzc.size()};
    for (int a = 0; a < 6; ++a) {
        *slots[a] = axes_ + off;
        off += lens[a];
    }
    ctx_.gf = GeomF{};
    if (p.geometry) geom_bind(ctx_.gf, axes_ + geo_off, p);
    ctx_.p.geometry = (int)p.geometry;
    ctx_.p.pow2 = p.geometry == 0 && pow2_grid(dxb, dyb, dzb, dxc, dyc, dzc, p.mu0, &ctx_.rc) ? 1 : 0;

    ctx_.p.gamma = p.gas_gamma;
    ctx_.p.mu0 = p.mu0;
    ctx_.p.visc1 = p.visc1;
    ctx_.p.visc2_norm = 0.25 * (p.gas_gamma + 1.0) * p.visc2;  // lagran.cpp:178
    ctx_.p.dt_multiplier = p.dt_multiplier;
    ctx_.p.eta_bg = p.eta_background;
    ctx_.p.eta0 = p.eta0;
    ctx_.p.j_max = p.j_max;
    ctx_.p.resistive = p.resistive_mhd ? 1 : 0;
    ctx_.p.rke = p.rke ? 1 : 0;

    if ((rc = check(cudaMalloc(&sc_, sizeof(Scalars)), "cudaMalloc(scalars)"))) return rc;
    Scalars s0{};
    s0.dt = 0.0;  // value-initialised runner data: the first step's viscosity sees dt = 0
    s0.dtmin_bits = 0x7FEFFFFFFFFFFFFFull;  // DBL_MAX
    if ((rc = check(cudaMemcpy(sc_, &s0, sizeof(s0), cudaMemcpyHostToDevice), "scalars upload"))) return rc;
    ctx_.sc = sc_;
    bytes_ = (long long)abytes + (long long)(packed.size() * sizeof(double)) + (long long)sizeof(Scalars);
    return check(cudaStreamSynchronize(stream_), "init sync");
}

int Solver::init_borrowed(const sams_lare_params &p, const sams_lare_bcs &bcs, const Ctx &ctx, int device,
                          cudaStream_t stream)
{
    if (p.geometry != 0) {
        err = "only Cartesian geometry is available on this entry point (no room for the metric tables)";
        return SAMS_ERR_UNSUPPORTED;
    }
    if (p.rke != 0) {
        err = "the remap kinetic-energy correction (rke) needs an array this entry point does not have";
        return SAMS_ERR_UNSUPPORTED;
    }
    p_ = p;
    device_ = device;
    {
        const long long n[3] = {p.nx, p.ny, p.nz};
        if (!bc_table_from(bc_, bcs, n, &err)) return SAMS_ERR_INVALID;
    }
    ctx_ = ctx;
    sc_ = ctx.sc;  // borrowed: release_borrowed() must clear it before destruction
    stream_ = stream;
    return check(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device), "sm count");
}

void Solver::release_borrowed()
{
    sc_ = nullptr;
    for (int f = 0; f < SAMS_NFIELDS; ++f) ctx_.f[f] = nullptr;
    for (int s = 0; s < NSCRATCH; ++s) ctx_.s[s] = nullptr;
}

int Solver::set_bc(int field, int dim, int edge, int kind, double value)
{
    if (field < 0 || field >= SAMS_NFIELDS || dim < 0 || dim > 2 || edge < 0 || edge > 1) {
        err = "invalid boundary-condition slot or kind";
        return SAMS_ERR_INVALID;
    }
    const long long n[3] = {p_.nx, p_.ny, p_.nz};
    BcTable t = bc_;
    if (!bc_slot_set(t, field, dim, edge, kind, value, n, &err)) return SAMS_ERR_INVALID;
    bc_ = t;
    for (auto &kv : graphs_) cudaGraphExecDestroy(kv.second);
    graphs_.clear();
    return SAMS_OK;
}

int Solver::set_stream(cudaStream_t s)
{
    stream_ = s ? s : own_stream_;
    for (auto &kv : graphs_) cudaGraphExecDestroy(kv.second);
    graphs_.clear();
    return SAMS_OK;
}

// Box rows are (nz+5) doubles; device rows are padded to g.sy with the row
// starting at offset zoff-2.  Copies from or to host memory go through a
// dense device staging buffer (one contiguous transfer at full link speed)
// and a repacking kernel; device-to-device copies are strided copies.
int Solver::staging(double **out)
{
    if (!staging_) {
        const size_t bytes = (size_t)(ctx_.g.nx + 5) * (ctx_.g.ny + 5) * (ctx_.g.nz + 5) * sizeof(double);
        int rc;
        if ((rc = check(cudaMalloc(&staging_, bytes), "cudaMalloc(staging)"))) return rc;
        bytes_ += (long long)bytes;
    }
    *out = staging_;
    return SAMS_OK;
}

int Solver::upload(int field, const double *src, cudaMemcpyKind kind)
{
    if (field < 0 || field >= SAMS_NFIELDS || !src) { err = "invalid field or buffer"; return SAMS_ERR_INVALID; }
    const Geom &g = ctx_.g;
    const size_t w = (size_t)(g.nz + 5) * sizeof(double);
    const size_t rows = (size_t)(g.nx + 5) * (size_t)(g.ny + 5);
    double *dst = ctx_.f[field] + (g.zoff - 2);
    if (kind == cudaMemcpyDeviceToDevice)
        return check(cudaMemcpy2DAsync(dst, (size_t)g.sy * sizeof(double), src, w, w, rows, kind, stream_), "upload");
    double *st;
    int rc;
    if ((rc = staging(&st))) return rc;
    if ((rc = check(cudaMemcpyAsync(st, src, w * rows, kind, stream_), "upload"))) return rc;
    k_repack<<<(unsigned)std::min<long long>(ceil_div((long long)(w / sizeof(double) * rows), kThreads), 8L * sm_count_),
               kThreads, 0, stream_>>>(st, ctx_.f[field], g, 1);
    return check(cudaGetLastError(), "repack");
}

int Solver::download(int field, double *dst, cudaMemcpyKind kind)
{
    if (field < 0 || field >= SAMS_NFIELDS || !dst) { err = "invalid field or buffer"; return SAMS_ERR_INVALID; }
    const Geom &g = ctx_.g;
    const size_t w = (size_t)(g.nz + 5) * sizeof(double);
    const size_t rows = (size_t)(g.nx + 5) * (size_t)(g.ny + 5);
    const double *src = ctx_.f[field] + (g.zoff - 2);
    int rc;
    if (kind == cudaMemcpyDeviceToDevice) {
        rc = check(cudaMemcpy2DAsync(dst, w, src, (size_t)g.sy * sizeof(double), w, rows, kind, stream_), "download");
    } else {
        double *st;
        if ((rc = staging(&st))) return rc;
        k_repack<<<(unsigned)std::min<long long>(ceil_div((long long)(w / sizeof(double) * rows), kThreads),
                                                 8L * sm_count_),
                   kThreads, 0, stream_>>>(ctx_.f[field], st, g, 0);
        if ((rc = check(cudaGetLastError(), "repack"))) return rc;
        rc = check(cudaMemcpyAsync(dst, st, w * rows, kind, stream_), "download");
    }
    if (rc) return rc;
    return check(cudaStreamSynchronize(stream_), "download sync");
}

// The x or y sweep's S6-S8 out of place into six scratch arrays free during
// the remap (the intermediates of the separate kernels live on chip here),
// then the solve's state pointers move to them; the y sweep writes back into
// the arrays the x sweep left, so after the two sweeps every pointer is
// where it started.
template <int DIR>
void Solver::launch_psweep(int ct_arg)
{
    static const int kOut[6] = {S_FX, S_FY, S_FZ, S_VH, S_FXV, S_FYV};
    static const int kState[6] = {SAMS_F_RHO, SAMS_F_ENERGY_ELECTRON, SAMS_F_ENERGY_ION,
                                  SAMS_F_VX, SAMS_F_VY, SAMS_F_VZ};
    const Geom &g = ctx_.g;
    const ops::SweepOut w{ctx_.s[kOut[0]], ctx_.s[kOut[1]], ctx_.s[kOut[2]],
                          ctx_.s[kOut[3]], ctx_.s[kOut[4]], ctx_.s[kOut[5]]};
    const int nd = DIR == 0 ? g.nx : g.ny, na = DIR == 0 ? g.ny : g.nx;
    const WinTile wt = march::win_tile(nd + 1, (long long)(na + 1) * (g.nz + 1), 3, 4 * sm_count_);
    const size_t smem = (size_t)ops::SweepFused<DIR>::NARR * ops::WinStore::P * ops::kWinK * sizeof(double);
    // rho1 (rho before the sweep) is rho itself here: the sweep writes the new
    // rho elsewhere (SweepVol skipped the copy)
    Ctx cc = ctx_;
    cc.s[S_R_RHO1] = ctx_.f[SAMS_F_RHO];
    if (ctx_.p.geometry)
        k_psweep<DIR, true><<<(unsigned)wt.blocks, ops::kWinThreads, smem, stream_>>>(cc, wt, w, ct_arg);
    else
        k_psweep<DIR, false><<<(unsigned)wt.blocks, ops::kWinThreads, smem, stream_>>>(cc, wt, w, ct_arg);
    ++launches_;
    // The points the sweep does not compute are ghost points of each array;
    // the fill that follows the sweep rewrites all of them from domain values
    // when every edge of these fields has a condition and every dimension at
    // least three cells (see enqueue_step).  Otherwise copy them over.
    if (!ghosts_refilled(FM_DENSITY | FM_ENERGY | FM_VELOCITY)) {
        const long long shell = BoxShell{{g.nx, g.ny, g.nz}, 1, 0}.count() + BoxShell{{g.nx, g.ny, g.nz}, 0, 0}.count();
        k_copy_shell<<<(unsigned)std::min<long long>(ceil_div(shell, kThreads), 8L * sm_count_), kThreads, 0,
                       stream_>>>(ctx_, w);
        ++launches_;
    }
    for (int q = 0; q < 6; ++q) std::swap(ctx_.f[kState[q]], ctx_.s[kOut[q]]);
}

// A cell op + node op pair (k_cellnode_march) over the whole box.
template <class P>
void Solver::launch_cellnode(int arg)
{
    const Geom &g = ctx_.g;
    const MarchTile m = march::march_tile(g.nz + 3, g.ny + 3, g.nx + 3, P::kMinBlocks * sm_count_);
    const size_t smem = (size_t)P::NR * 3 * kRP * sizeof(double);
    auto run = [&](auto kernel) { kernel<<<(unsigned)m.blocks, kMThreads, smem, stream_>>>(ctx_, m, arg); };
    const bool wide = march::march_wide(m);
    if (ctx_.p.geometry)
        run(k_cellnode_march<P, true, false, 0>);
    else if (ctx_.p.pow2)
        wide ? run(k_cellnode_march<P, false, true, march::kWideW>) : run(k_cellnode_march<P, false, true, 0>);
    else
        wide ? run(k_cellnode_march<P, false, false, march::kWideW>) : run(k_cellnode_march<P, false, false, 0>);
    ++launches_;
}

// The shock heating (k_heat_march) over cells 0..n+1.
void Solver::launch_heat()
{
    const Geom &g = ctx_.g;
    const MarchTile m = march::march_tile(g.nz + 2, g.ny + 2, g.nx + 2, march::kHeatMinBlocks * sm_count_);
    const size_t smem = (size_t)3 * 3 * kRP * sizeof(double);
    auto run = [&](auto kernel) { kernel<<<(unsigned)m.blocks, kMThreads, smem, stream_>>>(ctx_, m); };
    const bool wide = march::march_wide(m);
    if (ctx_.p.geometry)
        run(k_heat_march<true, false, 0>);
    else if (ctx_.p.pow2)
        wide ? run(k_heat_march<false, true, march::kWideW>) : run(k_heat_march<false, true, 0>);
    else
        wide ? run(k_heat_march<false, false, march::kWideW>) : run(k_heat_march<false, false, 0>);
    ++launches_;
}

// Pred1 + Pred2 fused (k_pred_march); the half-step pressures land in the
// S_CS / S_CSV arrays (free from here to the remap), whose slots then swap
// with S_PE / S_PI.
void Solver::launch_pred(int resistive)
{
    const Geom &g = ctx_.g;
    const MarchTile m = march::march_tile(g.nz + 1, g.ny + 1, g.nx + 1, 3 * sm_count_);
    const size_t smem = (size_t)march::PredRingSrc::NR * 3 * kRP * sizeof(double);
    double *pe = ctx_.s[S_CS], *pi = ctx_.s[S_CSV];
    auto run = [&](auto kernel) { kernel<<<(unsigned)m.blocks, kMThreads, smem, stream_>>>(ctx_, m, resistive, pe, pi); };
    const bool wide = march::march_wide(m);
    if (ctx_.p.geometry)
        run(k_pred_march<true, false, 0>);
    else if (ctx_.p.pow2)
        wide ? run(k_pred_march<false, true, march::kWideW>) : run(k_pred_march<false, true, 0>);
    else
        wide ? run(k_pred_march<false, false, march::kWideW>) : run(k_pred_march<false, false, 0>);
    ++launches_;
    std::swap(ctx_.s[S_PE], ctx_.s[S_CS]);
    std::swap(ctx_.s[S_PI], ctx_.s[S_CSV]);
}

// One resistive sub-step fused (k_resist_march); the new B goes to the
// S_CS / S_CSV / S_CV1 arrays (free during the sub-steps), whose slots then
// swap with the field's, so after the two sub-steps B is back in its own
// arrays and those three slots hold B as it was at the start of the last
// sub-step: the predictor's b1 (resistive_effects' copy, lagran.cpp:482-484).
void Solver::launch_resist(bool last)
{
    const Geom &g = ctx_.g;
    const MarchTile m = march::march_tile(g.nz + 5, g.ny + 5, g.nx + 5, 5 * sm_count_);
    const size_t smem = (size_t)ops::ResistRK::NOUT * 3 * kRP * sizeof(double);
    double *nb[3] = {ctx_.s[S_CS], ctx_.s[S_CSV], ctx_.s[S_CV1]};
    auto run = [&](auto kernel) { kernel<<<(unsigned)m.blocks, kMThreads, smem, stream_>>>(ctx_, m, nb[0], nb[1], nb[2]); };
    const bool wide = march::march_wide(m);
    if (ctx_.p.geometry)
        run(k_resist_march<true, false, 0>);
    else if (ctx_.p.pow2)
        wide ? run(k_resist_march<false, true, march::kWideW>) : run(k_resist_march<false, true, 0>);
    else
        wide ? run(k_resist_march<false, false, march::kWideW>) : run(k_resist_march<false, false, 0>);
    ++launches_;
    std::swap(ctx_.f[SAMS_F_BX], ctx_.s[S_CS]);
    std::swap(ctx_.f[SAMS_F_BY], ctx_.s[S_CSV]);
    std::swap(ctx_.f[SAMS_F_BZ], ctx_.s[S_CV1]);
    if (last) {
        std::swap(ctx_.s[S_B1X], ctx_.s[S_CS]);
        std::swap(ctx_.s[S_B1Y], ctx_.s[S_CSV]);
        std::swap(ctx_.s[S_B1Z], ctx_.s[S_CV1]);
    }
}

// SweepCT + SweepMass of one sweep (k_ctmass / k_ctmass_z).
template <int DIR>
bool Solver::launch_ctmass(int scale)
{
    const Geom &g = ctx_.g;
    // dm's periodic or zero-gradient fill along the sweep folded into the kernel (the slabs'
    // x fill is an exchange between slabs and stays)
    const int nd = DIR == 0 ? g.nx : (DIR == 1 ? g.ny : g.nz);
    int images = ops::kNoImages;
    if (!(halo_ && DIR == 0) && nd >= kBcSequentialBelow && bc_.kind[SAMS_F_DM][DIR][0] == bc_.kind[SAMS_F_DM][DIR][1]) {
        if (bc_.kind[SAMS_F_DM][DIR][0] == SAMS_BC_PERIODIC) images = ops::kPeriodicImages;
        if (bc_.kind[SAMS_F_DM][DIR][0] == SAMS_BC_ZERO_GRADIENT) images = ops::kCopyImages;
    }
    if (DIR == 2) {
        const ZTile z = march::z_tile(g.nz, (long long)(g.nx + 2) * (g.ny + 2));
        if (ctx_.p.geometry)
            k_ctmass_z<true><<<(unsigned)z.blocks, march::kZCtThreads, 0, stream_>>>(ctx_, z, images);
        else
            k_ctmass_z<false><<<(unsigned)z.blocks, march::kZCtThreads, 0, stream_>>>(ctx_, z, images);
    } else {
        const int na = DIR == 0 ? g.ny : g.nx;
        const WinTile w = march::win_tile(nd + 1, (long long)(na + 2) * (g.nz + 2), 3, 5 * sm_count_);
        const size_t smem = (size_t)ops::SweepCTMass<DIR>::NARR * march::kCtP * ops::kWinK * sizeof(double);
        if (ctx_.p.geometry)
            k_ctmass<DIR, true><<<(unsigned)w.blocks, ops::kWinThreads, smem, stream_>>>(ctx_, w, scale, images);
        else
            k_ctmass<DIR, false><<<(unsigned)w.blocks, ops::kWinThreads, smem, stream_>>>(ctx_, w, scale, images);
    }
    ++launches_;
    return images != ops::kNoImages;
}

template <class Op>
void Solver::launch(int arg)
{
    int lo[3], hi[3];
    Op::bounds(ctx_.g, arg, lo, hi);
    const long long plane = (long long)(hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1);
    dim3 grid((unsigned)ceil_div(plane, kThreads), (unsigned)(hi[0] - lo[0] + 1));
    if (ctx_.p.geometry)
        k_op<Op, true, false><<<grid, kThreads, 0, stream_>>>(ctx_, arg);
    else if (ctx_.p.pow2)
        k_op<Op, false, true><<<grid, kThreads, 0, stream_>>>(ctx_, arg);
    else
        k_op<Op, false, false><<<grid, kThreads, 0, stream_>>>(ctx_, arg);
    ++launches_;
}

// Whether a boundary fill of the fields in mask rewrites every ghost point
// from domain values, whatever the ghosts held before: every (dim, edge) of
// those fields has a condition (none is SAMS_BC_NONE), and every dimension
// has at least three cells (with fewer, an edge copy reads ghost planes it
// wrote).  Each condition reads domain planes of its own dimension; the fills
// run x, then y, then z, so a point that is a ghost in several dimensions
// ends with the value the last of them computes from the earlier ones.
bool Solver::ghosts_refilled(unsigned mask) const
{
    if (std::min(ctx_.g.nx, std::min(ctx_.g.ny, ctx_.g.nz)) < kBcSequentialBelow) return false;
    for (int f = 0; f < SAMS_NFIELDS; ++f)
        if (mask & (1u << f))
            for (int d = 0; d < 3; ++d)
                for (int e = 0; e < 2; ++e)
                    if (bc_.kind[f][d][e] == SAMS_BC_NONE) return false;
    return true;
}

bool Solver::all_periodic(unsigned mask) const
{
    for (int f = 0; f < SAMS_NFIELDS; ++f)
        if (mask & (1u << f))
            for (int d = 0; d < 3; ++d)
                for (int e = 0; e < 2; ++e)
                    if (bc_.kind[f][d][e] != SAMS_BC_PERIODIC) return false;
    return true;
}

template <unsigned MASK>
void Solver::bc_fill()
{
    constexpr unsigned mask = MASK;
    FieldList fl = make_list(mask);
    if (fl.n == 0) return;
    if (halo_) {  // a slab: x by exchange, then y and z in the same order as below
        halo_->fill_x(*this, mask);
        bc_fill_dim(mask, 1);
        bc_fill_dim(mask, 2);
        return;
    }
    const Geom &g = ctx_.g;
    // the one-pass gather needs every source inside the domain (n >= 3)
    if (all_periodic(mask) && std::min(g.nx, std::min(g.ny, g.nz)) >= kBcSequentialBelow) {
        const unsigned blocks = (unsigned)ceil_div(fill_points(g), kThreads);
        k_bc_periodic<MASK><<<blocks, kThreads, 0, stream_>>>(ctx_);
        ++launches_;
        return;
    }
    const int n[3] = {g.nx, g.ny, g.nz};
    bool compose = true;
    for (int q = 0; q < fl.n; ++q) compose = compose && bc_composable(bc_, fl.id[q], n);
    if (compose) {
        const long long e1 = g.ny + 5, e2 = g.nz + 5;
        const long long cnt = 6 * e1 * e2 + (long long)g.nx * 6 * e2 + (long long)g.nx * g.ny * 6;  // the largest shell
        dim3 grid((unsigned)ceil_div(cnt, kThreads), (unsigned)fl.n);
        k_bc_compose<<<grid, kThreads, 0, stream_>>>(ctx_, fl, bc_);
        ++launches_;
        return;
    }
    for (int d = 0; d < 3; ++d) bc_fill_dim(mask, d);
}

void Solver::bc_fill_dim(unsigned mask, int d)
{
    if (halo_ && d == 0) {
        halo_->fill_x(*this, mask);
        return;
    }
    for (int e = 0; e < 2; ++e) bc_fill_edge(mask, d, e);
}

void Solver::bc_fill_edge(unsigned mask, int d, int e)
{
    FieldList fl = make_list(mask);
    if (fl.n == 0) return;
    const Geom &g = ctx_.g;
    const long long ext[3] = {g.nx + 5, g.ny + 5, g.nz + 5};
    long long slab = 3;
    for (int q = 0; q < 3; ++q)
        if (q != d) slab *= ext[q];
    dim3 grid((unsigned)ceil_div(slab, kThreads), (unsigned)fl.n);
    k_bc_edge<<<grid, kThreads, 0, stream_>>>(ctx_, fl, bc_, d, e);
    ++launches_;
}

void Solver::enqueue_step(cudaEvent_t *marks)
{
    const int resistive = p_.resistive_mhd ? 1 : 0;
    auto mark = [&](int m) {
        if (marks) cudaEventRecord(marks[m], stream_);
    };
    mark(0);
    // ---- Lagrangian predictor ----
    launch_cellnode<PrepMarch>(resistive);
    launch<ops::Alpha>(0);
    {
        // Visc with two threads per cell (k_visc_split)
        int lo[3], hi[3];
        ops::Visc::bounds(ctx_.g, 0, lo, hi);
        const long long plane = (long long)(hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1);
        const int ni = hi[0] - lo[0] + 1;
        dim3 grid((unsigned)ceil_div(plane, kThreads / 2), (unsigned)(ni < 16 ? ni : 16));
        if (ctx_.p.geometry)
            k_visc_split<true, false><<<grid, kThreads, 0, stream_>>>(ctx_);
        else if (ctx_.p.pow2)
            k_visc_split<false, true><<<grid, kThreads, 0, stream_>>>(ctx_);
        else
            k_visc_split<false, false><<<grid, kThreads, 0, stream_>>>(ctx_);
        ++launches_;
    }
    if (halo_) halo_->reduce_dt(*this);
    k_dt_finalize<<<1, 1, 0, stream_>>>(sc_, p_.dt_multiplier, resistive);
    ++launches_;
    if (resistive) {
        for (int sub = 0; sub < 2; ++sub) {
            launch_resist(sub == 1);
            bc_fill<FM_BFIELD | FM_ENERGY>();
        }
    }
    launch_pred(resistive);
    bc_fill<FM_REMAPV>();
    mark(1);
    // ---- corrector ----
    // (Corr1 and Corr2 as one pass, with the velocities written out of place,
    // was measured slower on B200: Corr2 runs at 6 blocks per SM alone, at
    // Corr1's 2 when fused.)
    launch_heat();
    launch<ops::Corr2>(0);
    bc_fill<FM_VELOCITY | FM_ENERGY | FM_DENSITY>();
    mark(2);
    // ---- remap ----
    // B to and from flux form (BScale) folded into the x and z sweeps' CT
    // updates when the B fills rewrite every ghost point (ghosts_refilled):
    // the z sweep then unscales 0..n only, and the final B fill sets the
    // ghosts from those values, as it does after BScale's pass over the
    // whole box.
    const bool b_fill_all = ghosts_refilled(FM_BFIELD);
    const bool fused_xy = !p_.rke;  // k_psweep runs the x and y stages
    if (p_.rke) launch<ops::RkeZero>(0);
    if (!b_fill_all) launch<ops::BScale>(0);
    launch_cellnode<VolMarch<0>>(fused_xy ? 1 : 0);
    const bool dm_x = launch_ctmass<0>(b_fill_all ? 1 : 0);
    // The CT update changes only B, which the dm fill and the stages S6-S8
    // do not read, so the fused stages take it at their points 0..n (its
    // whole range; with the B scaling folded in, the fill after the sweep
    // writes B's ghosts from those points).
    if (!fused_xy) launch<ops::SweepCTUpd<0>>(b_fill_all ? 1 : 0);
    if (!dm_x) bc_fill_dim(FM_DM, 0);
    if (fused_xy) {
        launch_psweep<0>(b_fill_all ? 1 : 0);
    } else {
        launch<ops::SweepS6<0>>(0);
        launch<ops::SweepS7<0>>(0);
        if (p_.rke) {
            launch<ops::SweepRkeDk<0>>(0);
            launch<ops::SweepRkeGather<0>>(0);
        }
        launch<ops::SweepS8<0>>(0);
    }
    bc_fill<FM_ALL9>();
    mark(3);
    launch_cellnode<VolMarch<1>>(fused_xy ? 1 : 0);
    const bool dm_y = launch_ctmass<1>(0);
    if (!fused_xy) launch<ops::SweepCTUpd<1>>(0);
    if (!dm_y) bc_fill_dim(FM_DM, 1);
    if (fused_xy) {
        launch_psweep<1>(0);
    } else {
        launch<ops::SweepS6<1>>(0);
        launch<ops::SweepS7<1>>(0);
        if (p_.rke) {
            launch<ops::SweepRkeDk<1>>(0);
            launch<ops::SweepRkeGather<1>>(0);
        }
        launch<ops::SweepS8<1>>(0);
    }
    bc_fill<FM_ALL9>();
    mark(4);
    launch_cellnode<VolMarch<2>>(0);
    const bool dm_z = launch_ctmass<2>(0);
    const bool zfused = !p_.rke && ctx_.g.nz + 4 <= kZThreads;
    if (!zfused) launch<ops::SweepCTUpd<2>>(b_fill_all ? 2 : 0);
    if (!dm_z) bc_fill_dim(FM_DM, 2);
    if (zfused) {
        const Geom &g = ctx_.g;
        const int W = g.nz + 4, lines = kZThreads / W;
        const long long nl = (long long)(g.nx + 1) * (g.ny + 1);
        const size_t smem = (size_t)ops::SweepFused<2>::NARR * lines * W * sizeof(double);
        const unsigned blocks = (unsigned)ceil_div(nl, lines);
        const int ct_arg = b_fill_all ? 2 : 0;
        if (ctx_.p.geometry)
            k_zsweep<true><<<blocks, kZThreads, smem, stream_>>>(ctx_, ct_arg);
        else
            k_zsweep<false><<<blocks, kZThreads, smem, stream_>>>(ctx_, ct_arg);
        ++launches_;
    } else {
        launch<ops::SweepS6<2>>(0);
        launch<ops::SweepS7<2>>(0);
        if (p_.rke) {
            launch<ops::SweepRkeDk<2>>(0);
            launch<ops::SweepRkeGather<2>>(0);
        }
        launch<ops::SweepS8<2>>(0);
    }
    // with the B scaling folded into the z sweep's CT update, B needs no pass
    // of its own before the fill, so all nine fields take one fill (the fill
    // of each field is independent of the others')
    bc_fill<FM_ALL9>();
    if (!b_fill_all) {
        launch<ops::BScale>(1);
        bc_fill<FM_BFIELD>();
    }
    if (p_.rke) launch<ops::RkeEnergy>(0);  // after the remap (shared_data.h:414-417)
    mark(5);
}

int Solver::phase_times(double ms[5])
{
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    cudaEvent_t ev[6];
    for (int i = 0; i < 6; ++i)
        if ((rc = check(cudaEventCreate(&ev[i]), "cudaEventCreate"))) return rc;
    enqueue_step(ev);
    rc = check(cudaEventSynchronize(ev[5]), "phase sync");
    for (int i = 0; i < 5 && !rc; ++i) {
        float t = 0.f;
        rc = check(cudaEventElapsedTime(&t, ev[i], ev[i + 1]), "cudaEventElapsedTime");
        ms[i] = t;
    }
    for (int i = 0; i < 6; ++i) cudaEventDestroy(ev[i]);
    return rc;
}

int Solver::step(long long nsteps)
{
    if (nsteps < 0) { err = "negative step count"; return SAMS_ERR_INVALID; }
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    for (long long s = 0; s < nsteps; ++s) {
        long long before = launches_;
        enqueue_step();
        launches_per_step_ = launches_ - before;
        if ((rc = check(cudaGetLastError(), "step launch"))) return rc;
    }
    return SAMS_OK;
}

int Solver::step_graph(long long nsteps)
{
    if (nsteps < 0) { err = "negative step count"; return SAMS_ERR_INVALID; }
    if (nsteps == 0) return SAMS_OK;
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    auto it = graphs_.find(nsteps);
    if (it == graphs_.end()) {
        cudaGraph_t graph;
        if ((rc = check(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal), "begin capture"))) return rc;
        for (long long s = 0; s < nsteps; ++s) {
            long long before = launches_;
            enqueue_step();
            launches_per_step_ = launches_ - before;
        }
        if ((rc = check(cudaStreamEndCapture(stream_, &graph), "end capture"))) return rc;
        cudaGraphExec_t exec;
        rc = check(cudaGraphInstantiate(&exec, graph, 0), "graph instantiate");
        cudaGraphDestroy(graph);
        if (rc) return rc;
        it = graphs_.emplace(nsteps, exec).first;
    }
    return check(cudaGraphLaunch(it->second, stream_), "graph launch");
}

int Solver::sync()
{
    int rc = check(cudaStreamSynchronize(stream_), "synchronize");
    if (rc) return rc;
    Scalars s;
    if ((rc = scalars(s))) return rc;
    if (s.status) {
        err = "the CFL timestep became non-finite or non-positive";
        return SAMS_ERR_NONFINITE;
    }
    return SAMS_OK;
}

int Solver::set_scalars(double dt, double time, long long step)
{
    Scalars h{};
    h.dt = dt;
    h.dtr = dt;
    h.time = time;
    h.step = step;
    const double big = DBL_MAX;
    std::memcpy(&h.dtmin_bits, &big, sizeof big);
    int rc = check(cudaMemcpyAsync(sc_, &h, sizeof(Scalars), cudaMemcpyHostToDevice, stream_), "scalars write");
    if (rc) return rc;
    return check(cudaStreamSynchronize(stream_), "scalars sync");
}

int Solver::scalars(Scalars &out)
{
    int rc = check(cudaMemcpyAsync(&out, sc_, sizeof(Scalars), cudaMemcpyDeviceToHost, stream_), "scalars read");
    if (rc) return rc;
    return check(cudaStreamSynchronize(stream_), "scalars sync");
}

}  // namespace sams
