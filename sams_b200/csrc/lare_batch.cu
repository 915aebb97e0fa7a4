// lare_batch.cu -- batched LARE3D solves (see lare_batch.cuh).
//
// The per-point work is the same sams::ops code as the single-solve path;
// what changes is the launcher: a persistent grid strides over a worklist of
// tiles from every live solve, loading each tile's solve context (pointers,
// geometry, parameters) into shared memory.  The fused kernels run the same
// bodies as the single solve's (lare_march.cuh), their worklist the blocks of
// every solve's own tiling; boundary fills walk the ghost shells of all
// solves.  One batched step is the same phase sequence as
// Solver::enqueue_step, each phase a single launch for the whole batch.
#include "lare_batch.cuh"
#include "lare_ops.cuh"
#include "lare_march.cuh"
#include "lare_bc.cuh"
#include "lare_geom_host.h"
#include "lare_repack.cuh"

#include <algorithm>
#include <cstring>

namespace sams {

namespace {

constexpr int kT = 256;
constexpr int kFillPoints = kT;  // shell points per entry of the fill's block list

// Where the x and y sweeps write the six state fields (launch_psweep of the
// single solve), and those fields.
__constant__ const int kSweepOut[6] = {S_FX, S_FY, S_FZ, S_VH, S_FXV, S_FYV};

// Whether field f's own range holds the point and has it as a ghost.
__device__ __forceinline__ bool field_ghost(const Geom &g, int f, int q0, int q1, int q2)
{
    const int q[3] = {q0, q1, q2}, n[3] = {g.nx, g.ny, g.nz};
    bool ghost = false;
    for (int d = 0; d < 3; ++d) {
        const int h = field_half(f, d);
        if (q[d] < (h ? -2 : -1)) return false;
        ghost = ghost || q[d] <= 0 || q[d] > n[d] - h;
    }
    return ghost;
}

template <class T>
__device__ __forceinline__ void load_words(T &dst, const T *src)
{
    const int nw = (int)(sizeof(T) / sizeof(int));
    const int *s = reinterpret_cast<const int *>(src);
    int *d = reinterpret_cast<int *>(&dst);
    for (int w = threadIdx.x; w < nw; w += blockDim.x) d[w] = s[w];
}

// GEO: some solve of the batch is curvilinear (the Cartesian instantiation,
// used when none is, carries no metric factors).
template <class Op, bool GEO, bool P2>
__global__ void __launch_bounds__(kT, (MinBlocksBatch<Op, P2>::value))
    kb_op(const Ctx *__restrict__ ctxs, const Tile *__restrict__ tiles, int ntiles, int arg, int tile_i)
{
    __shared__ Ctx c;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const Tile tl = tiles[t];
        // threads walk the op's own (j, k) range (no idle lanes on the ghost
        // planes of thin solves); the tiles cover the whole box plane, so
        // every op's range is inside them, and a tile past the op's range
        // is skipped before its context is staged (uniform over the block)
        const Ctx *src = ctxs + tl.inst;
        int lo[3], hi[3];
        Op::bounds(src->g, arg, lo, hi);
        const int nk = hi[2] - lo[2] + 1;
        if (tl.p0 >= (hi[1] - lo[1] + 1) * nk || tl.i0 > hi[0] || tl.i0 + tile_i - 1 < lo[0]) continue;
        __syncthreads();
        load_words(c, src);
        __syncthreads();
        const int p = tl.p0 + (int)threadIdx.x;
        if (p >= (hi[1] - lo[1] + 1) * nk) continue;
        const int j = lo[1] + p / nk, k = lo[2] + p % nk;
        const int ia = max(tl.i0, lo[0]), ib = min(tl.i0 + tile_i - 1, hi[0]);
        for (int i = ia; i <= ib; ++i) Op::template run<GEO, P2>(c, arg, i, j, k);
    }
}

template <bool GEO, bool P2>
__global__ void __launch_bounds__(kT, 4)  // tuned on n x n x 4 solves; k_visc_split has 3
    kb_visc(const Ctx *__restrict__ ctxs, const Tile *__restrict__ tiles, int ntiles, int tile_i)
{
    __shared__ Ctx c;
    __shared__ double wmin[kT / 32];
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const Tile tl = tiles[t];
        int lo[3], hi[3];
        ops::Visc::bounds(ctxs[tl.inst].g, 0, lo, hi);
        const int nk = hi[2] - lo[2] + 1;
        if (tl.p0 >= (hi[1] - lo[1] + 1) * nk || tl.i0 > hi[0] || tl.i0 + tile_i - 1 < lo[0]) continue;
        __syncthreads();
        load_words(c, ctxs + tl.inst);
        __syncthreads();
        // two threads per cell, as the single-solve k_visc_split: warps 0-3
        // run the heating and forces, warps 4-7 the viscous pressure and CFL
        // candidate, each over the tile's points in two rounds of 128
        const int half = (int)threadIdx.x >> 7;
        double best = DBL_MAX;
        bool bad = false;
        for (int r = 0; r < 2; ++r) {
            const int p = tl.p0 + r * (kT / 2) + ((int)threadIdx.x & (kT / 2 - 1));
            if (p >= (hi[1] - lo[1] + 1) * nk) continue;
            const int j = lo[1] + p / nk, k = lo[2] + p % nk;
            const int ia = max(tl.i0, lo[0]), ib = min(tl.i0 + tile_i - 1, hi[0]);
            for (int i = ia; i <= ib; ++i) {
                if (half == 0)
                    ops::Visc::template heat_forces<GEO, P2>(c, i, j, k, bad);
                else if (i <= c.g.nx && j <= c.g.ny && k <= c.g.nz)
                    best = dev::pmin(best, ops::Visc::template cfl<GEO, P2>(c, i, j, k, bad));
            }
        }
        if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&c.sc->status, 1);
        for (int off = 16; off > 0; off >>= 1) best = dev::pmin(best, __shfl_xor_sync(0xffffffffu, best, off));
        if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            double m = wmin[0];
            for (int w = 1; w < kT / 32; ++w) m = dev::pmin(m, wmin[w]);
            if (m < DBL_MAX) atomicMin(&c.sc->dtmin_bits, (unsigned long long)__double_as_longlong(m));
        }
    }
}

// The fused phases (bodies in lare_march.cuh) over every live solve's blocks:
// a persistent grid strides over the phase's block list, staging each block's
// solve context and tilings in shared memory.
struct BlockScratch {
    Ctx c;
    SolveTiles t;
};
template <class F>
__device__ __forceinline__ void for_blocks(const Ctx *ctxs, const SolveTiles *st, const BlockRef *blocks, int n, F &&run)
{
    __shared__ BlockScratch sh;
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const BlockRef r = blocks[q];
        __syncthreads();
        load_words(sh.c, ctxs + r.inst);
        load_words(sh.t, st + r.inst);
        __syncthreads();
        run(sh.c, sh.t, r.block);
    }
}

#define KB_ARGS const Ctx *__restrict__ ctxs, const SolveTiles *__restrict__ st, const BlockRef *__restrict__ blocks, int n

template <class P, bool GEO, bool P2>
__global__ void __launch_bounds__(march::kMThreads, P::kMinBlocks) kb_cellnode(KB_ARGS, int arg)
{
    extern __shared__ double ring[];
    for_blocks(ctxs, st, blocks, n, [&](const Ctx &c, const SolveTiles &t, int b) {
        march::cellnode<P, GEO, P2>(c, t.cellnode, b, arg >= 0 ? arg : c.p.resistive, ring);
    });
}

template <bool GEO, bool P2>
__global__ void __launch_bounds__(march::kMThreads, 3) kb_pred(KB_ARGS)
{
    extern __shared__ double ring[];
    for_blocks(ctxs, st, blocks, n, [&](const Ctx &c, const SolveTiles &t, int b) {
        march::pred<GEO, P2>(c, t.pred, b, c.p.resistive, c.s[S_CS], c.s[S_CSV], ring);
    });
}

template <bool GEO, bool P2>
__global__ void __launch_bounds__(march::kMThreads, march::kHeatMinBlocks) kb_heat(KB_ARGS)
{
    extern __shared__ double ring[];
    for_blocks(ctxs, st, blocks, n,
               [&](const Ctx &c, const SolveTiles &t, int b) { march::heat_edges<GEO, P2>(c, t.heat, b, ring); });
}

template <bool GEO, bool P2>
__global__ void __launch_bounds__(march::kMThreads, 5) kb_resist(KB_ARGS)
{
    extern __shared__ double ring[];
    for_blocks(ctxs, st, blocks, n, [&](const Ctx &c, const SolveTiles &t, int b) {
        march::resist<GEO, P2>(c, t.resist, b, c.s[S_CS], c.s[S_CSV], c.s[S_CV1], ring);
    });
}

template <int DIR, bool GEO>
__global__ void __launch_bounds__(ops::kWinThreads, 5) kb_ctmass(KB_ARGS, int scale)
{
    extern __shared__ double csm[];
    for_blocks(ctxs, st, blocks, n, [&](const Ctx &c, const SolveTiles &t, int b) {
        march::ctmass<DIR, GEO>(c, t.ct[DIR], b, scale, t.images[DIR], csm);
    });
}

template <bool GEO>
__global__ void __launch_bounds__(march::kZCtThreads, 4) kb_ctmass_z(KB_ARGS)
{
    __shared__ double zsm[ops::SweepCTMass<2>::NARR * march::kZCtThreads];
    for_blocks(ctxs, st, blocks, n,
               [&](const Ctx &c, const SolveTiles &t, int b) { march::ctmass_z<GEO>(c, t.ctz, b, t.images[2], zsm); });
}

template <int DIR, bool GEO>
__global__ void __launch_bounds__(ops::kWinThreads, 4) kb_psweep(KB_ARGS, int ct_arg)
{
    extern __shared__ double psm[];
    for_blocks(ctxs, st, blocks, n, [&](const Ctx &c, const SolveTiles &t, int b) {
        const ops::SweepOut w{c.s[kSweepOut[0]], c.s[kSweepOut[1]], c.s[kSweepOut[2]],
                              c.s[kSweepOut[3]], c.s[kSweepOut[4]], c.s[kSweepOut[5]]};
        march::psweep<DIR, GEO>(c, t.stage[DIR], b, w, ct_arg, psm);
    });
}

template <bool GEO>
__global__ void __launch_bounds__(march::kZThreads, 4) kb_zsweep(KB_ARGS, int ct_arg)
{
    extern __shared__ double zsm[];
    for_blocks(ctxs, st, blocks, n,
               [&](const Ctx &c, const SolveTiles &, int b) { march::zsweep<GEO>(c, b, ct_arg, zsm); });
}
#undef KB_ARGS

// The ghost points of the out-of-place sweeps' arrays that no fill rewrites
// (k_copy_shell of the single solve), for the solves that need it.
__global__ void __launch_bounds__(kT) kb_copy_shell(const Ctx *__restrict__ ctxs, const SolveTiles *__restrict__ st,
                                                    const int *__restrict__ live, int nlive)
{
    for (int li = blockIdx.y; li < nlive; li += gridDim.y) {
        const int inst = live[li];
        if (st[inst].refilled) continue;
        const Ctx &c = ctxs[inst];
        const Geom g = c.g;
        const ops::SweepOut w{c.s[kSweepOut[0]], c.s[kSweepOut[1]], c.s[kSweepOut[2]],
                              c.s[kSweepOut[3]], c.s[kSweepOut[4]], c.s[kSweepOut[5]]};
        ops::copy_shell(c, g, w, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
    }
}

// Per-solve CFL finalisation (the single-solve k_dt_finalize, one thread per
// live solve).
__global__ void kb_dt_finalize(const Ctx *__restrict__ ctxs, const int *__restrict__ live, int nlive)
{
    const int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= nlive) return;
    const Ctx &c = ctxs[live[li]];
    Scalars *sc = c.sc;
    double m = __longlong_as_double((long long)sc->dtmin_bits);
    double dt = c.p.dt_multiplier * m;
    sc->dtr = dt;
    dt = dt < DBL_MAX ? dt : DBL_MAX;
    sc->dt = dt;
    if (c.p.resistive) {
        int nsub = (int)(dt / sc->dtr) + 1;
        sc->nsub = nsub;
        sc->dt_sub = dt / (double)nsub;
    }
    sc->dtmin_bits = (unsigned long long)__double_as_longlong(DBL_MAX);
    if (!(m < DBL_MAX) || !(dt > 0.0) || !(dt < DBL_MAX)) sc->status = 1;
    sc->time += dt;
    sc->step += 1;
}

__device__ __forceinline__ int locate(const long long *off, int n, long long g)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Boundary fill of the fields in `mask` for every live solve whose conditions
// on them can be applied in one pass (SolveTiles::periodic: the composite
// periodic gather of k_bc_periodic; SolveTiles::compose: bc_compose_value).
// Each entry of the list is kFillPoints consecutive points of one solve's
// ghost shell: its whole box -2..n+2 outside 1..n (1..n-1: the half-cell
// fields' index n is a ghost too), x slabs, then y slabs inside x, then z
// slabs inside x and y.  A point is decomposed once and then written for every
// field in whose own range it is a ghost, one field after another (all loads
// first, as periodic_copy has them, was 3% slower here).
__global__ void __launch_bounds__(kT) kb_bc_fill(const Ctx *__restrict__ ctxs, const SolveTiles *__restrict__ st,
                                                 const BcTable *__restrict__ bcs, const BlockRef *__restrict__ blocks, int n,
                                                 unsigned mask, int resistive_only)
{
    for (int b = blockIdx.x; b < n; b += gridDim.x) {
        const BlockRef r = blocks[b];
        const Ctx &c = ctxs[r.inst];
        const bool periodic = (mask & ~st[r.inst].periodic) == 0;
        if (!periodic && (mask & ~st[r.inst].compose) != 0) continue;  // edge by edge (kb_bc_edge)
        if (resistive_only && !c.p.resistive) continue;
        const Geom &g = c.g;
        int q0, q1, q2;
        if (!fill_point(g, r.block * kFillPoints + (int)threadIdx.x, q0, q1, q2)) continue;
        if (periodic) {
            const int s0 = q0 <= 0 ? q0 + g.nx : (q0 > g.nx ? q0 - g.nx : q0);
            const int s1 = q1 <= 0 ? q1 + g.ny : (q1 > g.ny ? q1 - g.ny : q1);
            const int s2 = q2 <= 0 ? q2 + g.nz : (q2 > g.nz ? q2 - g.nz : q2);
            const int dst = box_off(g, q0, q1, q2), src = box_off(g, s0, s1, s2);
            if (dst == src) continue;  // (an index n that is no ghost of a centred field, and keeps its value in a half-cell one)
            for (int f = 0; f < SAMS_NFIELDS; ++f) {
                if (!(mask & (1u << f))) continue;
                // centred dimensions start at -1
                if ((q0 < -1 && !field_half(f, 0)) || (q1 < -1 && !field_half(f, 1)) || (q2 < -1 && !field_half(f, 2)))
                    continue;
                double *a = c.f[f];
                a[dst] = a[src];
            }
            continue;
        }
        const BcTable &bt = bcs[r.inst];
        for (int f = 0; f < SAMS_NFIELDS; ++f) {
            if (!(mask & (1u << f)) || !field_ghost(g, f, q0, q1, q2)) continue;
            double *a = c.f[f];
            const double v = bc_compose_value<2>(a, g, bt, f, q0, q1, q2);
            a[box_off(g, q0, q1, q2)] = v;
        }
    }
}

// One (dimension, edge) of the fields in `mask` for every live solve (those
// the one-pass fill, or for dm the CT + mass kernels, have done are skipped);
// the point formula and the ordering rule of small dimensions are lare_bc.cuh's.
__global__ void kb_bc_edge(const Ctx *__restrict__ ctxs, const SolveTiles *__restrict__ st,
                           const BcTable *__restrict__ bcs, const int *__restrict__ live,
                           const long long *__restrict__ off, int nlive, long long total, unsigned mask, int d, int e,
                           int dm_only, int resistive_only)
{
    for (long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x; gi < total;
         gi += (long long)gridDim.x * blockDim.x) {
        const int li = locate(off, nlive, gi);
        const int inst = live[li];
        // handled by the CT + mass kernels (dm) or the one-pass fill
        if (dm_only ? st[inst].images[d] != ops::kNoImages
                    : (mask & ~st[inst].periodic) == 0 || (mask & ~st[inst].compose) == 0)
            continue;
        const Ctx &c = ctxs[inst];
        if (resistive_only && !c.p.resistive) continue;
        const BcTable &bt = bcs[inst];
        const long long t = gi - off[li];
        const Geom &g = c.g;
        for (int f = 0; f < SAMS_NFIELDS; ++f) {
            if (!(mask & (1u << f))) continue;
            const int kind = bt.kind[f][d][e];
            if (kind == SAMS_BC_NONE) continue;
            const BcEdge sl = bc_edge_slab(g, f, d, e);
            const int e1 = sl.hi[1] - sl.lo[1] + 1, e2 = sl.hi[2] - sl.lo[2] + 1;
            if (t >= (long long)(sl.hi[0] - sl.lo[0] + 1) * e1 * e2) continue;
            int q[3];
            q[0] = sl.lo[0] + (int)(t / ((long long)e1 * e2));
            q[1] = sl.lo[1] + (int)((t / e2) % e1);
            q[2] = sl.lo[2] + (int)(t % e2);
            bc_edge_apply(c.f[f], g, sl, bt, f, d, e, q);
        }
    }
}

void axes_host(double lo, double hi, long long n, std::vector<double> &db, std::vector<double> &dc)
{
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

Geom batch_geom(const sams_lare_params &p)
{
    Geom g{};
    g.nx = (int)p.nx;
    g.ny = (int)p.ny;
    g.nz = (int)p.nz;
    if (p.nz >= 32) {  // long rows: pad to 8 doubles with interior k = 1 on a 32-byte boundary
        g.zoff = 3;
        g.sy = (int)(((p.nz + 6) + 7) / 8 * 8);
    } else {            // short rows (e.g. nz = 4): dense
        g.zoff = 2;
        g.sy = (int)(p.nz + 5);
    }
    g.sx = (int)((p.ny + 5) * g.sy);
    g.nelem = (p.nx + 5) * (long long)g.sx;
    return g;
}

long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

}  // namespace

// ---------------------------------------------------------------------------

Batch::~Batch()
{
    cudaSetDevice(device_);
    drop_graphs();
    for (auto &s : slots_) free_slot(s);
    cudaFree(d_tables_);
    if (own_stream_) cudaStreamDestroy(own_stream_);
}

int Batch::check(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return SAMS_OK;
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? SAMS_ERR_NOMEM : SAMS_ERR_CUDA;
}

void Batch::drop_graphs()
{
    for (auto &kv : graphs_) cudaGraphExecDestroy(kv.second);
    graphs_.clear();
}

void Batch::free_slot(BatchSlot &s)
{
    if (s.arena) cudaFree(s.arena);
    if (s.axes) cudaFree(s.axes);
    if (s.sc) cudaFree(s.sc);
    s = BatchSlot{};
}

int Batch::init(int device)
{
    device_ = device;
    int rc;
    if ((rc = check(cudaSetDevice(device), "cudaSetDevice"))) return rc;
    if ((rc = check(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking), "cudaStreamCreate"))) return rc;
    stream_ = own_stream_;
    cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device);
    return SAMS_OK;
}

int Batch::set_stream(cudaStream_t s)
{
    stream_ = s ? s : own_stream_;
    drop_graphs();
    return SAMS_OK;
}

long long Batch::bytes_for(const sams_lare_params &p)
{
    Geom g = batch_geom(p);
    return (long long)(SAMS_NFIELDS + NSCRATCH + (p.rke ? 1 : 0)) * g.nelem * 8 + 8 * 2 * (p.nx + p.ny + p.nz + 18) + 256 +
           (p.geometry ? 8LL * (long long)geom_table_size(p) : 0LL);
}

int Batch::add(const sams_lare_params &p, const sams_lare_bcs &bcs, int *id)
{
    if (p.nx < 1 || p.ny < 1 || p.nz < 1 || p.nx > 60000 || p.ny > 60000 || p.nz > 60000) {
        err = "grid sizes must be in 1..60000";
        return SAMS_ERR_INVALID;
    }
    if (p.geometry < 0 || p.geometry > 2) { err = "geometry must be 0 (Cartesian), 1 (cylindrical) or 2 (spherical)"; return SAMS_ERR_UNSUPPORTED; }
    if (!(p.x_max > p.x_min) || !(p.y_max > p.y_min) || !(p.z_max > p.z_min)) { err = "empty domain"; return SAMS_ERR_INVALID; }
    {
        // tile planes and ghost shells are indexed with 32-bit integers
        const long long e1 = p.ny + 5, e2 = p.nz + 5;
        const long long shell = 5 * e1 * e2 + p.nx * 5 * e2 + p.nx * p.ny * 5;
        const long long rows = (p.nz >= 32 ? ((p.nz + 6) + 7) / 8 * 8 : e2) * e1 * (p.nx + 5);
        if (rows > INT32_MAX || shell > INT32_MAX) {
            err = "one array or the ghost shell of this solve exceeds 2^31 points";
            return SAMS_ERR_UNSUPPORTED;
        }
    }
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    BatchSlot s;
    s.p = p;
    {
        const long long n[3] = {p.nx, p.ny, p.nz};
        if (!bc_table_from(s.bc, bcs, n, &err)) return SAMS_ERR_INVALID;
    }
    Geom g = batch_geom(p);
    const size_t abytes = (size_t)(SAMS_NFIELDS + NSCRATCH + (p.rke ? 1 : 0)) * (size_t)g.nelem * sizeof(double);
    if ((rc = check(cudaMalloc(&s.arena, abytes), "cudaMalloc(solve)"))) return rc;
    cudaMemsetAsync(s.arena, 0, abytes, stream_);
    std::vector<double> dxb, dyb, dzb, dxc, dyc, dzc;
    axes_host(p.x_min, p.x_max, p.nx, dxb, dxc);
    axes_host(p.y_min, p.y_max, p.ny, dyb, dyc);
    axes_host(p.z_min, p.z_max, p.nz, dzb, dzc);
    std::vector<double> packed;
    for (auto *v : {&dxb, &dyb, &dzb, &dxc, &dyc, &dzc}) packed.insert(packed.end(), v->begin(), v->end());
    const size_t geo_off = packed.size();
    if (p.geometry) {  // metric factors after the spacings
        std::vector<double> t = geom_tables(p);
        packed.insert(packed.end(), t.begin(), t.end());
    }
    if ((rc = check(cudaMalloc(&s.axes, packed.size() * sizeof(double)), "cudaMalloc(axes)"))) { free_slot(s); return rc; }
    if ((rc = check(cudaMemcpy(s.axes, packed.data(), packed.size() * sizeof(double), cudaMemcpyHostToDevice), "axes"))) {
        free_slot(s);
        return rc;
    }
    if ((rc = check(cudaMalloc(&s.sc, sizeof(Scalars)), "cudaMalloc(scalars)"))) { free_slot(s); return rc; }
    Scalars s0{};
    s0.dtmin_bits = 0x7FEFFFFFFFFFFFFFull;
    if ((rc = check(cudaMemcpy(s.sc, &s0, sizeof(s0), cudaMemcpyHostToDevice), "scalars"))) { free_slot(s); return rc; }
    Ctx &c = s.ctx;
    c.g = g;
    for (int f = 0; f < SAMS_NFIELDS; ++f) c.f[f] = s.arena + (size_t)f * g.nelem;
    for (int q = 0; q < NSCRATCH; ++q) c.s[q] = s.arena + (size_t)(SAMS_NFIELDS + q) * g.nelem;
    c.dke = p.rke ? s.arena + (size_t)(SAMS_NFIELDS + NSCRATCH) * g.nelem : nullptr;
    size_t o = 0;
    const double **slots[6] = {&c.ax.dxb, &c.ax.dyb, &c.ax.dzb, &c.ax.dxc, &c.ax.dyc, &c.ax.dzc};
    const size_t lens[6] = {dxb.size(), dyb.size(), dzb.size(), dxc.size(), dyc.size(), dzc.size()};
    for (int a = 0; a < 6; ++a) {
        *slots[a] = s.axes + o;
        o += lens[a];
    }
    c.gf = GeomF{};
    if (p.geometry) geom_bind(c.gf, s.axes + geo_off, p);
    c.p.geometry = (int)p.geometry;
    c.p.pow2 = p.geometry == 0 && pow2_grid(dxb, dyb, dzb, dxc, dyc, dzc, p.mu0, &c.rc) ? 1 : 0;
    c.p.gamma = p.gas_gamma;
    c.p.mu0 = p.mu0;
    c.p.visc1 = p.visc1;
    c.p.visc2_norm = 0.25 * (p.gas_gamma + 1.0) * p.visc2;
    c.p.dt_multiplier = p.dt_multiplier;
    c.p.eta_bg = p.eta_background;
    c.p.eta0 = p.eta0;
    c.p.j_max = p.j_max;
    c.p.resistive = p.resistive_mhd ? 1 : 0;
    c.p.rke = p.rke ? 1 : 0;
    c.sc = s.sc;
    s.bytes = (long long)abytes + (long long)(packed.size() * sizeof(double)) + (long long)sizeof(Scalars);
    s.live = true;
    int slot = -1;
    for (size_t q = 0; q < slots_.size(); ++q)
        if (!slots_[q].live) { slot = (int)q; break; }
    if (slot < 0) {
        slot = (int)slots_.size();
        slots_.push_back(BatchSlot{});
    }
    slots_[slot] = s;
    *id = slot;
    dirty_ = true;
    drop_graphs();
    return check(cudaStreamSynchronize(stream_), "add sync");
}

int Batch::remove(int id)
{
    if (id < 0 || id >= (int)slots_.size() || !slots_[id].live) { err = "no such solve"; return SAMS_ERR_INVALID; }
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    if ((rc = check(cudaStreamSynchronize(stream_), "remove sync"))) return rc;
    free_slot(slots_[id]);
    dirty_ = true;
    drop_graphs();
    return SAMS_OK;
}

// Host boxes are dense.  So are the rows of short-row solves, and one
// contiguous copy moves a field; padded rows go through a repacking kernel
// and the solve's first scratch array, which nothing reads between steps.
// (Copied row by row, a 64^3 solve's 13 fields took 12.5 ms in and its nine
// results 6.7 ms out, against 2.7 and 1.6 through the single solve's
// contiguous copies.)
static bool dense(const Geom &g) { return g.sy == g.nz + 5 && g.zoff == 2; }
unsigned Batch::repack_grid(const Geom &g) const
{
    return (unsigned)std::min<long long>(ceil_div((long long)(g.nx + 5) * (g.ny + 5) * (g.nz + 5), kT), 8L * sm_count_);
}

int Batch::upload(int id, int field, const double *src, cudaMemcpyKind kind)
{
    if (id < 0 || id >= (int)slots_.size() || !slots_[id].live || field < 0 || field >= SAMS_NFIELDS || !src) {
        err = "invalid solve, field or buffer";
        return SAMS_ERR_INVALID;
    }
    const Geom &g = slots_[id].ctx.g;
    const Ctx &c = slots_[id].ctx;
    const size_t bytes = (size_t)(g.nx + 5) * (g.ny + 5) * (g.nz + 5) * sizeof(double);
    if (dense(g)) return check(cudaMemcpyAsync(c.f[field], src, bytes, kind, stream_), "upload");
    double *box = c.s[0];
    int rc;
    if ((rc = check(cudaMemcpyAsync(box, src, bytes, kind, stream_), "upload"))) return rc;
    k_repack<<<repack_grid(g), kT, 0, stream_>>>(box, c.f[field], g, 1);
    return check(cudaGetLastError(), "repack");
}

int Batch::download_async(int id, int field, double *dst)
{
    if (id < 0 || id >= (int)slots_.size() || !slots_[id].live || field < 0 || field >= SAMS_NFIELDS || !dst) {
        err = "invalid solve, field or buffer";
        return SAMS_ERR_INVALID;
    }
    const Geom &g = slots_[id].ctx.g;
    const Ctx &c = slots_[id].ctx;
    const size_t bytes = (size_t)(g.nx + 5) * (g.ny + 5) * (g.nz + 5) * sizeof(double);
    const double *from = c.f[field];
    if (!dense(g)) {
        double *box = c.s[0];
        k_repack<<<repack_grid(g), kT, 0, stream_>>>(c.f[field], box, g, 0);
        int rc;
        if ((rc = check(cudaGetLastError(), "repack"))) return rc;
        from = box;
    }
    return check(cudaMemcpyAsync(dst, from, bytes, cudaMemcpyDefault, stream_), "download");
}

int Batch::download(int id, int field, double *dst, cudaMemcpyKind kind)
{
    (void)kind;
    int rc = download_async(id, field, dst);
    if (rc) return rc;
    return check(cudaStreamSynchronize(stream_), "download sync");
}

// How one solve's phases are cut into blocks and its conditions met.  share:
// the part of the device that this solve's blocks can count on.
static SolveTiles solve_tiles(const BatchSlot &s, double share, int sm_count)
{
    SolveTiles t{};
    const Geom &g = s.ctx.g;
    auto sm = [&](int per_sm) { return std::max(1, (int)(share * per_sm * sm_count)); };
    t.cellnode = march::march_tile(g.nz + 3, g.ny + 3, g.nx + 3, sm(march::PrepMarch::kMinBlocks));
    t.pred = march::march_tile(g.nz + 1, g.ny + 1, g.nx + 1, sm(3));
    t.heat = march::march_tile(g.nz + 2, g.ny + 2, g.nx + 2, sm(march::kHeatMinBlocks));
    t.resist = march::march_tile(g.nz + 5, g.ny + 5, g.nx + 5, sm(5));
    for (int d = 0; d < 2; ++d) {
        const int nd = d == 0 ? g.nx : g.ny, na = d == 0 ? g.ny : g.nx;
        t.ct[d] = march::win_tile(nd + 1, (long long)(na + 2) * (g.nz + 2), 3, sm(5));
        t.stage[d] = march::win_tile(nd + 1, (long long)(na + 1) * (g.nz + 1), 3, sm(4));
    }
    t.ctz = march::z_tile(g.nz, (long long)(g.nx + 2) * (g.ny + 2));
    const int n[3] = {g.nx, g.ny, g.nz};
    const bool three = std::min(n[0], std::min(n[1], n[2])) >= kBcSequentialBelow;
    t.refilled = three ? 1 : 0;
    t.b_refilled = three ? 1 : 0;
    for (int f = 0; f < SAMS_NFIELDS; ++f) {
        bool per = three, none = false;
        for (int d = 0; d < 3; ++d)
            for (int e = 0; e < 2; ++e) {
                per = per && s.bc.kind[f][d][e] == SAMS_BC_PERIODIC;
                none = none || s.bc.kind[f][d][e] == SAMS_BC_NONE;
            }
        if (per) t.periodic |= 1u << f;
        if (bc_composable(s.bc, f, n)) t.compose |= 1u << f;
        // (ghosts_refilled of the single solve)
        if (none && ((1u << f) & (FM_DENSITY | FM_ENERGY | FM_VELOCITY))) t.refilled = 0;
        if (none && ((1u << f) & FM_BFIELD)) t.b_refilled = 0;
    }
    for (int d = 0; d < 3; ++d) {
        const int l = s.bc.kind[SAMS_F_DM][d][0], u = s.bc.kind[SAMS_F_DM][d][1];
        if (n[d] < kBcSequentialBelow || l != u) continue;
        if (l == SAMS_BC_PERIODIC) t.images[d] = ops::kPeriodicImages;
        if (l == SAMS_BC_ZERO_GRADIENT) t.images[d] = ops::kCopyImages;
    }
    return t;
}

// The contexts of one solve through a step: scratch arrays and fields trade
// places after the out-of-place phases exactly as Solver's launches swap them.
static void solve_contexts(const Ctx &base, bool fused_xy, Ctx out[Batch::NCTX])
{
    Ctx c = base;
    out[Batch::C_START] = c;
    auto resist_swap = [&] {
        std::swap(c.f[SAMS_F_BX], c.s[S_CS]);
        std::swap(c.f[SAMS_F_BY], c.s[S_CSV]);
        std::swap(c.f[SAMS_F_BZ], c.s[S_CV1]);
    };
    if (c.p.resistive) resist_swap();
    out[Batch::C_SUB] = c;
    if (c.p.resistive) {
        resist_swap();
        std::swap(c.s[S_B1X], c.s[S_CS]);
        std::swap(c.s[S_B1Y], c.s[S_CSV]);
        std::swap(c.s[S_B1Z], c.s[S_CV1]);
    }
    out[Batch::C_PRED] = c;
    std::swap(c.s[S_PE], c.s[S_CS]);
    std::swap(c.s[S_PI], c.s[S_CSV]);
    out[Batch::C_REMAP] = c;
    // the out-of-place sweeps read rho itself as rho1
    static const int kOut[6] = {S_FX, S_FY, S_FZ, S_VH, S_FXV, S_FYV};
    static const int kState[6] = {SAMS_F_RHO, SAMS_F_ENERGY_ELECTRON, SAMS_F_ENERGY_ION, SAMS_F_VX, SAMS_F_VY, SAMS_F_VZ};
    out[Batch::C_X] = c;
    if (fused_xy) {
        out[Batch::C_X].s[S_R_RHO1] = c.f[SAMS_F_RHO];
        for (int q = 0; q < 6; ++q) std::swap(c.f[kState[q]], c.s[kOut[q]]);
    }
    out[Batch::C_Y] = c;
    if (fused_xy) out[Batch::C_Y].s[S_R_RHO1] = c.f[SAMS_F_RHO];
}

int Batch::rebuild()
{
    const size_t nslot = std::max<size_t>(slots_.size(), 1);
    std::vector<Ctx> ctx(NCTX * nslot);
    std::vector<BcTable> bcs(nslot);
    std::vector<SolveTiles> st(nslot);
    std::vector<int> live;
    std::vector<long long> slab_off[3];
    std::vector<Tile> tiles;
    std::vector<BlockRef> lists[NPHASE];
    long long slab[3] = {0, 0, 0};
    has_resistive_ = has_rke_ = has_geo_ = 0;
    all_pow2_ = 1;
    fold_ = true;
    shell_ = edges_ = 0;
    dm_edges_[0] = dm_edges_[1] = dm_edges_[2] = false;
    zfuse_ = true;
    double cells = 0.0;
    long long elems = 0;
    for (auto &s : slots_) {
        if (!s.live) continue;
        elems += s.ctx.g.nelem;
        has_rke_ |= s.ctx.p.rke;
        if (s.ctx.g.nz + 4 > march::kZThreads) zfuse_ = false;
        cells += (double)(s.p.nx + 5) * (double)(s.p.ny + 5) * (double)(s.p.nz + 5);
    }
    fused_xy_ = !has_rke_;
    zfuse_ = zfuse_ && !has_rke_;
    for (size_t q = 0; q < slots_.size(); ++q) {
        BatchSlot &s = slots_[q];
        if (!s.live) continue;
        bcs[q] = s.bc;
        Ctx cs[NCTX];
        Ctx base = s.ctx;
        base.g.far = far_from_l2(elems);
        solve_contexts(base, fused_xy_, cs);
        for (int v = 0; v < NCTX; ++v) ctx[(size_t)v * nslot + q] = cs[v];
        const Geom &g = s.ctx.g;
        const double share = (double)(s.p.nx + 5) * (double)(s.p.ny + 5) * (double)(s.p.nz + 5) / cells;
        const SolveTiles t = st[q] = solve_tiles(s, share, sm_count_);
        live.push_back((int)q);
        has_resistive_ |= s.ctx.p.resistive;
        has_geo_ |= s.ctx.p.geometry != 0;
        all_pow2_ &= s.ctx.p.pow2;
        fold_ = fold_ && t.b_refilled;
        if (!t.refilled) shell_ = 1;
        for (unsigned m : {(unsigned)FM_REMAPV, (unsigned)FM_ALL9})  // (every mask that bc_fill takes is part of one of these)
            if ((m & ~t.periodic) && (m & ~t.compose)) edges_ = 1;
        const long long e0 = g.nx + 5, e1 = g.ny + 5, e2 = g.nz + 5;
        for (int d = 0; d < 3; ++d) {
            slab_off[d].push_back(slab[d]);
            if (t.images[d] == ops::kNoImages) dm_edges_[d] = true;
        }
        slab[0] += 3 * e1 * e2;
        slab[1] += 3 * e0 * e2;
        slab[2] += 3 * e0 * e1;
        const int plane = (int)(e1 * e2);
        for (int i0 = -2; i0 <= g.nx + 2; i0 += tile_i_)
            for (int p0 = 0; p0 < plane; p0 += kT) tiles.push_back(Tile{(int)q, i0, p0, 0});
        auto blocks = [&](int phase, long long n) {
            for (long long b = 0; b < n; ++b) lists[phase].push_back(BlockRef{(int)q, (int)b});
        };
        blocks(P_CELLNODE, t.cellnode.blocks);
        if (s.ctx.p.resistive) blocks(P_RESIST, t.resist.blocks);
        blocks(P_PRED, t.pred.blocks);
        blocks(P_HEAT, t.heat.blocks);
        blocks(P_CTX, t.ct[0].blocks);
        blocks(P_CTY, t.ct[1].blocks);
        blocks(P_CTZ, t.ctz.blocks);
        blocks(P_STX, t.stage[0].blocks);
        blocks(P_STY, t.stage[1].blocks);
        if (zfuse_) {
            const int lines = march::kZThreads / (g.nz + 4);
            blocks(P_STZ, ceil_div((long long)(g.nx + 1) * (g.ny + 1), lines));
        }
        blocks(P_FILL, ceil_div(fill_points(g), kFillPoints));
    }
    nlive_ = (int)live.size();
    ntiles_ = (int)tiles.size();
    for (int d = 0; d < 3; ++d) slab_total_[d] = slab[d];
    // one device buffer for all tables
    size_t off = 0;
    auto place = [&](size_t bytes) {
        const size_t at = off;
        off += (std::max<size_t>(bytes, 16) + 15) / 16 * 16;
        return at;
    };
    const size_t o_ctx = place(ctx.size() * sizeof(Ctx)), o_bc = place(bcs.size() * sizeof(BcTable));
    const size_t o_st = place(st.size() * sizeof(SolveTiles)), o_tiles = place(tiles.size() * sizeof(Tile));
    const size_t o_live = place(live.size() * sizeof(int));
    const size_t o_slab = place(3 * live.size() * sizeof(long long));
    size_t o_list[NPHASE];
    for (int ph = 0; ph < NPHASE; ++ph) o_list[ph] = place(lists[ph].size() * sizeof(BlockRef));
    int rc;
    if (off > table_cap_bytes_) {
        cudaFree(d_tables_);
        d_tables_ = nullptr;
        table_cap_bytes_ = 0;
        const size_t cap = off * 2;
        if ((rc = check(cudaMalloc((void **)&d_tables_, cap), "cudaMalloc(batch tables)"))) return rc;
        table_cap_bytes_ = cap;
    }
    std::vector<char> host(off);
    auto put = [&](size_t at, const void *src, size_t n) { if (n) std::memcpy(host.data() + at, src, n); };
    put(o_ctx, ctx.data(), ctx.size() * sizeof(Ctx));
    put(o_bc, bcs.data(), bcs.size() * sizeof(BcTable));
    put(o_st, st.data(), st.size() * sizeof(SolveTiles));
    put(o_tiles, tiles.data(), tiles.size() * sizeof(Tile));
    put(o_live, live.data(), live.size() * sizeof(int));
    for (int d = 0; d < 3; ++d) put(o_slab + d * live.size() * sizeof(long long), slab_off[d].data(), live.size() * sizeof(long long));
    for (int v = 0; v < NCTX; ++v) d_ctx_[v] = reinterpret_cast<Ctx *>(d_tables_ + o_ctx) + (size_t)v * nslot;
    d_bc_ = reinterpret_cast<BcTable *>(d_tables_ + o_bc);
    d_st_ = reinterpret_cast<SolveTiles *>(d_tables_ + o_st);
    d_tiles_ = reinterpret_cast<Tile *>(d_tables_ + o_tiles);
    d_live_ = reinterpret_cast<int *>(d_tables_ + o_live);
    d_slab_off_ = reinterpret_cast<long long *>(d_tables_ + o_slab);
    for (int ph = 0; ph < NPHASE; ++ph) {
        put(o_list[ph], lists[ph].data(), lists[ph].size() * sizeof(BlockRef));
        d_list_[ph] = reinterpret_cast<BlockRef *>(d_tables_ + o_list[ph]);
        nlist_[ph] = (int)lists[ph].size();
    }
    if ((rc = check(cudaMemcpyAsync(d_tables_, host.data(), off, cudaMemcpyHostToDevice, stream_), "batch tables"))) return rc;
    dirty_ = false;
    // keep the host-side copy alive until the async copy is done
    return check(cudaStreamSynchronize(stream_), "batch tables sync");
}

template <class Op>
void Batch::launch(int ctx, int arg)
{
    if (ntiles_ == 0) return;
    const int grid = std::min(ntiles_, sm_count_ * blocks_per_sm_);
    if (has_geo_)
        kb_op<Op, true, false><<<grid, kT, 0, stream_>>>(d_ctx_[ctx], d_tiles_, ntiles_, arg, tile_i_);
    else if (all_pow2_)
        kb_op<Op, false, true><<<grid, kT, 0, stream_>>>(d_ctx_[ctx], d_tiles_, ntiles_, arg, tile_i_);
    else
        kb_op<Op, false, false><<<grid, kT, 0, stream_>>>(d_ctx_[ctx], d_tiles_, ntiles_, arg, tile_i_);
}

void Batch::launch_visc()
{
    if (ntiles_ == 0) return;
    const int grid = std::min(ntiles_, sm_count_ * blocks_per_sm_);
    const Ctx *c = d_ctx_[C_START];
    if (has_geo_)
        kb_visc<true, false><<<grid, kT, 0, stream_>>>(c, d_tiles_, ntiles_, tile_i_);
    else if (all_pow2_)
        kb_visc<false, true><<<grid, kT, 0, stream_>>>(c, d_tiles_, ntiles_, tile_i_);
    else
        kb_visc<false, false><<<grid, kT, 0, stream_>>>(c, d_tiles_, ntiles_, tile_i_);
}

// A fused phase over its block list: `per_sm` blocks per SM (the kernel's
// register cap), each striding over the list.
#define FUSED_ARGS d_ctx_[ctx], d_st_, d_list_[ph], nlist_[ph]
#define FUSED_LAUNCH(kernel, per_sm, threads, smem, ...)                                                            \
    if (nlist_[ph]) kernel<<<std::min(nlist_[ph], sm_count_ * (per_sm)), threads, smem, stream_>>>(FUSED_ARGS, ##__VA_ARGS__)
#define FUSED_GP(kernel, per_sm, smem, ...)                                                                         \
    if (has_geo_) { FUSED_LAUNCH((kernel<true, false>), per_sm, march::kMThreads, smem, ##__VA_ARGS__); }           \
    else if (all_pow2_) { FUSED_LAUNCH((kernel<false, true>), per_sm, march::kMThreads, smem, ##__VA_ARGS__); }     \
    else { FUSED_LAUNCH((kernel<false, false>), per_sm, march::kMThreads, smem, ##__VA_ARGS__); }

constexpr size_t kPlaneBytes = 3 * march::kRP * sizeof(double);  // one ring array

template <class P>
void Batch::launch_cellnode(int ctx, int arg)
{
    const int ph = P_CELLNODE;
    const size_t smem = P::NR * kPlaneBytes;
    if (has_geo_) { FUSED_LAUNCH((kb_cellnode<P, true, false>), P::kMinBlocks, march::kMThreads, smem, arg); }
    else if (all_pow2_) { FUSED_LAUNCH((kb_cellnode<P, false, true>), P::kMinBlocks, march::kMThreads, smem, arg); }
    else { FUSED_LAUNCH((kb_cellnode<P, false, false>), P::kMinBlocks, march::kMThreads, smem, arg); }
}

void Batch::launch_resist(int ctx)
{
    const int ph = P_RESIST;
    FUSED_GP(kb_resist, 5, ops::ResistRK::NOUT * kPlaneBytes);
}

void Batch::launch_pred(int ctx)
{
    const int ph = P_PRED;
    FUSED_GP(kb_pred, 3, march::PredRingSrc::NR * kPlaneBytes);
}

void Batch::launch_heat(int ctx)
{
    const int ph = P_HEAT;
    FUSED_GP(kb_heat, march::kHeatMinBlocks, 3 * kPlaneBytes);
}

template <int DIR>
void Batch::launch_ctmass(int ctx, int scale)
{
    const int ph = DIR == 0 ? P_CTX : (DIR == 1 ? P_CTY : P_CTZ);
    if constexpr (DIR == 2) {
        (void)scale;
        if (has_geo_) { FUSED_LAUNCH(kb_ctmass_z<true>, 4, march::kZCtThreads, 0); }
        else { FUSED_LAUNCH(kb_ctmass_z<false>, 4, march::kZCtThreads, 0); }
    } else {
        const size_t smem = (size_t)ops::SweepCTMass<DIR>::NARR * march::kCtP * ops::kWinK * sizeof(double);
        if (has_geo_) { FUSED_LAUNCH((kb_ctmass<DIR, true>), 5, ops::kWinThreads, smem, scale); }
        else { FUSED_LAUNCH((kb_ctmass<DIR, false>), 5, ops::kWinThreads, smem, scale); }
    }
    if (dm_edges_[DIR]) bc_edges(ctx, FM_DM, DIR, true, false);
}

template <int DIR>
void Batch::launch_psweep(int ctx, int ct_arg)
{
    const int ph = DIR == 0 ? P_STX : P_STY;
    const size_t smem = (size_t)ops::SweepFused<DIR>::NARR * ops::WinStore::P * ops::kWinK * sizeof(double);
    if (has_geo_) { FUSED_LAUNCH((kb_psweep<DIR, true>), 4, ops::kWinThreads, smem, ct_arg); }
    else { FUSED_LAUNCH((kb_psweep<DIR, false>), 4, ops::kWinThreads, smem, ct_arg); }
    if (shell_) kb_copy_shell<<<dim3(64, (unsigned)std::min(nlive_, 1024)), kT, 0, stream_>>>(d_ctx_[ctx], d_st_, d_live_, nlive_);
}

void Batch::launch_zsweep(int ctx, int ct_arg)
{
    const int ph = P_STZ;
    const size_t smem = (size_t)ops::SweepFused<2>::NARR * march::kZThreads * sizeof(double);
    if (has_geo_) { FUSED_LAUNCH(kb_zsweep<true>, 4, march::kZThreads, smem, ct_arg); }
    else { FUSED_LAUNCH(kb_zsweep<false>, 4, march::kZThreads, smem, ct_arg); }
}

void Batch::bc_edges(int ctx, unsigned mask, int d, bool dm_only, bool resistive_only)
{
    const int g2 = (int)std::min<long long>(ceil_div(slab_total_[d], kT), (long long)sm_count_ * 8);
    for (int e = 0; e < 2; ++e)
        kb_bc_edge<<<g2, kT, 0, stream_>>>(d_ctx_[ctx], d_st_, d_bc_, d_live_, d_slab_off_ + (size_t)d * nlive_, nlive_,
                                           slab_total_[d], mask, d, e, dm_only ? 1 : 0, resistive_only ? 1 : 0);
}

void Batch::bc_fill(int ctx, unsigned mask, bool resistive_only)
{
    if (nlive_ == 0) return;
    const int n = nlist_[P_FILL];
    kb_bc_fill<<<std::min(n, sm_count_ * 8), kT, 0, stream_>>>(d_ctx_[ctx], d_st_, d_bc_, d_list_[P_FILL], n, mask,
                                                               resistive_only ? 1 : 0);
    if (edges_)
        for (int d = 0; d < 3; ++d) bc_edges(ctx, mask, d, false, resistive_only);
}

// The same phases in the same order as Solver::enqueue_step.
void Batch::enqueue_step()
{
    if (nlive_ == 0) return;
    // ---- Lagrangian predictor ----
    launch_cellnode<march::PrepMarch>(C_START, -1);
    launch<ops::Alpha>(C_START, 0);
    launch_visc();
    kb_dt_finalize<<<(unsigned)ceil_div(nlive_, 128), 128, 0, stream_>>>(d_ctx_[C_START], d_live_, nlive_);
    if (has_resistive_) {
        launch_resist(C_START);
        bc_fill(C_SUB, FM_BFIELD | FM_ENERGY, true);
        launch_resist(C_SUB);
        bc_fill(C_PRED, FM_BFIELD | FM_ENERGY, true);
    }
    launch_pred(C_PRED);
    bc_fill(C_REMAP, FM_REMAPV, false);
    // ---- corrector ----
    launch_heat(C_REMAP);
    launch<ops::Corr2>(C_REMAP, 0);
    bc_fill(C_REMAP, FM_VELOCITY | FM_ENERGY | FM_DENSITY, false);
    // ---- remap ----
    if (has_rke_) launch<ops::RkeZero>(C_REMAP, 0);
    if (!fold_) launch<ops::BScale>(C_REMAP, 0);
    launch_cellnode<march::VolMarch<0>>(C_X, fused_xy_ ? 1 : 0);
    launch_ctmass<0>(C_X, fold_ ? 1 : 0);
    stages<0>(C_X, fold_ ? 1 : 0);
    bc_fill(C_Y, FM_ALL9, false);
    launch_cellnode<march::VolMarch<1>>(C_Y, fused_xy_ ? 1 : 0);
    launch_ctmass<1>(C_Y, 0);
    stages<1>(C_Y, 0);
    bc_fill(C_REMAP, FM_ALL9, false);
    launch_cellnode<march::VolMarch<2>>(C_REMAP, 0);
    launch_ctmass<2>(C_REMAP, 0);
    stages<2>(C_REMAP, fold_ ? 2 : 0);
    bc_fill(C_REMAP, FM_ALL9, false);
    if (!fold_) {
        launch<ops::BScale>(C_REMAP, 1);
        bc_fill(C_REMAP, FM_BFIELD, false);
    }
    if (has_rke_) launch<ops::RkeEnergy>(C_REMAP, 0);
}

// The CT update and S6-S8 of one sweep: one kernel, or the separate ones.
template <int DIR>
void Batch::stages(int ctx, int ct_arg)
{
    if constexpr (DIR == 2) {
        if (zfuse_) return launch_zsweep(ctx, ct_arg);
    } else {
        if (fused_xy_) return launch_psweep<DIR>(ctx, ct_arg);
    }
    launch<ops::SweepCTUpd<DIR>>(ctx, ct_arg);
    launch<ops::SweepS6<DIR>>(ctx, 0);
    launch<ops::SweepS7<DIR>>(ctx, 0);
    if (has_rke_) {  // solves without rke return at once (Phys::rke)
        launch<ops::SweepRkeDk<DIR>>(ctx, 0);
        launch<ops::SweepRkeGather<DIR>>(ctx, 0);
    }
    launch<ops::SweepS8<DIR>>(ctx, 0);
}

int Batch::step(long long nsteps)
{
    if (nsteps < 0) { err = "negative step count"; return SAMS_ERR_INVALID; }
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    if (dirty_ && (rc = rebuild())) return rc;
    for (long long s = 0; s < nsteps; ++s) enqueue_step();
    return check(cudaGetLastError(), "batch step launch");
}

int Batch::step_graph(long long nsteps)
{
    if (nsteps < 0) { err = "negative step count"; return SAMS_ERR_INVALID; }
    if (nsteps == 0) return SAMS_OK;
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    if (dirty_) {
        if ((rc = rebuild())) return rc;
        drop_graphs();
    }
    auto it = graphs_.find(nsteps);
    if (it == graphs_.end()) {
        cudaGraph_t graph;
        if ((rc = check(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal), "begin capture"))) return rc;
        for (long long s = 0; s < nsteps; ++s) enqueue_step();
        if ((rc = check(cudaStreamEndCapture(stream_, &graph), "end capture"))) return rc;
        cudaGraphExec_t exec;
        rc = check(cudaGraphInstantiate(&exec, graph, 0), "graph instantiate");
        cudaGraphDestroy(graph);
        if (rc) return rc;
        it = graphs_.emplace(nsteps, exec).first;
    }
    return check(cudaGraphLaunch(it->second, stream_), "graph launch");
}

int Batch::sync() { return check(cudaStreamSynchronize(stream_), "batch synchronize"); }

int Batch::scalars(int id, Scalars &out)
{
    if (id < 0 || id >= (int)slots_.size() || !slots_[id].live) { err = "no such solve"; return SAMS_ERR_INVALID; }
    int rc = check(cudaMemcpyAsync(&out, slots_[id].sc, sizeof(Scalars), cudaMemcpyDeviceToHost, stream_), "scalars");
    if (rc) return rc;
    return check(cudaStreamSynchronize(stream_), "scalars sync");
}

int Batch::set_tuning(int tile_i, int blocks_per_sm)
{
    if (tile_i < 1 || tile_i > 64 || blocks_per_sm < 1 || blocks_per_sm > 32) {
        err = "tile_i must be 1..64 and blocks_per_sm 1..32";
        return SAMS_ERR_INVALID;
    }
    tile_i_ = tile_i;
    blocks_per_sm_ = blocks_per_sm;
    dirty_ = true;
    drop_graphs();
    return SAMS_OK;
}

// Time every candidate tiling on the live batch for trial_steps steps and keep
// the fastest.  The state of every solve (13 fields and its scalars) is
// copied aside first and restored afterwards, so tuning leaves the solves
// exactly where they were.
int Batch::autotune(int trial_steps, int *tile_i, int *blocks_per_sm, double *best_ms)
{
    if (trial_steps < 1) trial_steps = 1;
    int rc;
    if ((rc = check(cudaSetDevice(device_), "cudaSetDevice"))) return rc;
    std::vector<double *> backup;
    std::vector<Scalars *> sback;
    for (auto &s : slots_) {
        if (!s.live) { backup.push_back(nullptr); sback.push_back(nullptr); continue; }
        double *b = nullptr;
        Scalars *sb = nullptr;
        size_t n = (size_t)SAMS_NFIELDS * (size_t)s.ctx.g.nelem * sizeof(double);
        if ((rc = check(cudaMalloc(&b, n), "cudaMalloc(autotune backup)"))) break;
        if ((rc = check(cudaMalloc(&sb, sizeof(Scalars)), "cudaMalloc(autotune backup)"))) { cudaFree(b); break; }
        cudaMemcpyAsync(b, s.arena, n, cudaMemcpyDeviceToDevice, stream_);
        cudaMemcpyAsync(sb, s.sc, sizeof(Scalars), cudaMemcpyDeviceToDevice, stream_);
        backup.push_back(b);
        sback.push_back(sb);
    }
    const int tiles[] = {1, 2, 4, 8};
    const int bps[] = {2, 4, 8};
    int bt = tile_i_, bb = blocks_per_sm_;
    double best = 1e300;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (int ti : tiles) {
        if (rc) break;
        for (int b : bps) {
            set_tuning(ti, b);
            if ((rc = step(1))) break;  // warm-up (also rebuilds the tables)
            cudaEventRecord(e0, stream_);
            if ((rc = step(trial_steps))) break;
            cudaEventRecord(e1, stream_);
            if ((rc = check(cudaEventSynchronize(e1), "autotune sync"))) break;
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                bt = ti;
                bb = b;
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    for (size_t q = 0; q < slots_.size(); ++q) {
        if (!slots_[q].live || !backup[q]) continue;
        size_t n = (size_t)SAMS_NFIELDS * (size_t)slots_[q].ctx.g.nelem * sizeof(double);
        cudaMemcpyAsync(slots_[q].arena, backup[q], n, cudaMemcpyDeviceToDevice, stream_);
        cudaMemcpyAsync(slots_[q].sc, sback[q], sizeof(Scalars), cudaMemcpyDeviceToDevice, stream_);
    }
    cudaStreamSynchronize(stream_);
    for (auto *b : backup) cudaFree(b);
    for (auto *b : sback) cudaFree(b);
    set_tuning(bt, bb);
    if (tile_i) *tile_i = bt;
    if (blocks_per_sm) *blocks_per_sm = bb;
    if (best_ms) *best_ms = best / trial_steps;
    return rc;
}

long long Batch::device_bytes() const
{
    long long b = (long long)table_cap_bytes_;
    for (auto &s : slots_)
        if (s.live) b += s.bytes;
    return b;
}

int Batch::live_count() const
{
    int n = 0;
    for (auto &s : slots_) n += s.live ? 1 : 0;
    return n;
}

long long Batch::live_cells() const
{
    long long n = 0;
    for (auto &s : slots_)
        if (s.live) n += s.p.nx * s.p.ny * s.p.nz;
    return n;
}

}  // namespace sams
