// lare_march.cuh -- the fused kernels' bodies, shared by the single-solve
// launcher (lare_solver.cu: one grid per solve) and the batched one
// (lare_batch.cu: one grid over the blocks of many solves).  Each body runs
// block b of one solve's phase with the solve's context c:
//   march kernels   a producer op feeding a consumer op through a ring of
//                   planes in shared memory, marching along x
//   window kernels  CT + mass fluxes and the stages S6-S8 over windows along
//                   the sweep
#pragma once

#include "lare_ops.cuh"

namespace sams {
namespace march {

// Shape of a march kernel's blocks: the ring plane is W x R cells (W along z,
// one per thread), of which (W - 1) x (R - 1) are the block's own points; a
// block walks MI planes along x.
struct MarchTile {
    int W, R, MI;
    int nkt, njt;  // tiles along z and y
    int blocks;    // nkt * njt * chunks
};
constexpr int kMThreads = 288;
constexpr int kRP = kMThreads;  // ring plane stride

// The tile of a phase whose own points are nk x nj x ni.  A plane costs as
// many blocks as it has tiles, so W is the width with the fewest of them
// (288 = W x R cells, the halo row and column recomputed), weighed by the row
// pieces a warp's 32 lanes cover: at W = 32 a warp is one row, at W = 26 it
// touches parts of two or three and a block took 11% (predictor) to 26%
// (shock heating) longer at 256^3.  32 x 9 suits long rows; rows of 5 to 70
// values (n x n x 4 solves, 32^3 cubes, 512 x 256 x 64) leave up to six lanes
// of seven idle with it (a 512 x 256 x 64 step took 10.1 ms, 8.4 with these
// tiles; a 128 x 128 x 4 one 222 us, 192; a 32^3 one 79 us, 62).  MI trades the
// plane that each chunk produces twice against blocks in flight: 16 planes
// where that gives every SM its blocks four times over, else the number that
// the whole waves of blocks take the least time with.
inline MarchTile march_tile(int nk, int nj, int ni, int sm_blocks)
{
    MarchTile best{};
    double cost = 0.0;
    for (int W = 2; W <= 96; ++W) {
        const int R = kMThreads / W;
        if (W > nk + 1 && W > 2) break;
        const int bk = (nk + W - 2) / (W - 1), bj = (nj + R - 2) / (R - 1);
        const double pieces = 32 % W == 0 ? 32.0 / W : (W % 32 == 0 ? 1.0 : 1.0 + 31.0 / W);
        const double c = (double)bk * bj * (1.0 + 0.12 * (pieces - 1.0));
        if (best.W == 0 || c < cost) {
            best.W = W;
            best.R = R;
            best.nkt = bk;
            best.njt = bj;
            cost = c;
        }
    }
    const long long plane = (long long)best.nkt * best.njt;
    best.MI = 16;
    if (plane * ((ni + 15) / 16) < 4LL * sm_blocks) {
        double tbest = 0.0;
        for (int MI = 16; MI >= 1; --MI) {
            const long long waves = (plane * ((ni + MI - 1) / MI) + sm_blocks - 1) / sm_blocks;
            const double t = (double)waves * (MI + 0.5);
            if (tbest == 0.0 || t < tbest) {
                best.MI = MI;
                tbest = t;
            }
        }
    }
    best.blocks = (int)(plane * ((ni + best.MI - 1) / best.MI));
    return best;
}

// The 32 x 9 tile of long rows as compile-time constants (CW = 32; CW = 0
// takes the tile's own): ring offsets fold into the addresses, which is 6 to
// 9% of the predictor's and the resistive march's time at 256^3.
constexpr int kWideW = 32, kWideR = kMThreads / kWideW;
inline bool march_wide(const MarchTile &m) { return m.W == kWideW; }

// Block b's tile: own points from (i0, j0, k0) (relative to the phase's first
// point), planes i0..i0+ni-1 where the chunk is not cut off by the range.
struct MarchAt {
    int i0, j0, k0;
    int pj, pk;   // the thread's ring cell
    bool cell;    // it has one
    bool own;     // ... of the block's own points
};
template <int CW = 0>
__host__ __device__ __forceinline__ MarchAt march_at(const MarchTile &m, int b, int t)
{
    const int W = CW ? CW : m.W, R = CW ? kMThreads / (CW ? CW : 1) : m.R;
    MarchAt a;
    const int tk = b % m.nkt;
    b /= m.nkt;
    const int tj = b % m.njt;
    a.i0 = (b / m.njt) * m.MI;
    a.k0 = tk * (W - 1);
    a.j0 = tj * (R - 1);
    a.pj = t / W;
    a.pk = t - a.pj * W;
    a.cell = a.pj < R;
    a.own = a.pj < R - 1 && a.pk < W - 1;
    return a;
}

// Ask L2 for the line at offset o of an array (no register waits for it).
// These kernels wait on memory first (8 to 16 of the 14 to 24 cycles between
// a warp's instructions), and where the arrays outgrow L2 half of those waits
// go to DRAM, one after another as each stage reaches its arrays.  So each
// block asks at its start, or a plane ahead, for what its later stages read:
// 256^3 x and y stages 1.33 -> 1.24 and 1.47 -> 1.36 ms, predictor 1.52 -> 1.46,
// resistive sub-step 0.41 -> 0.37, heating 0.46 -> 0.42.  On grids that stay in
// L2 (96^3) the cell-to-node marches lost 7% with it: Geom::far draws the line
// at twelve arrays, what a phase reads, against L2's 126 MB.  (Asking for the
// next wave's block instead was 4% slower over the step than none at all.)
__device__ __forceinline__ void prefetch(const double *a, int o) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a + o)); }

struct RingSrc {
    const double *ring;
    __device__ double operator()(int arr, int q) const { return ring[arr * 3 * kRP + q]; }
};
// The predictor's ring: Pred1's outputs with p_e + p_i in the PE slot (Pred2
// reads only that sum), five arrays.
struct PredRingSrc {
    static constexpr int NR = ops::Pred1::PI;  // CV1, B1X, B1Y, B1Z, PE (= p_e + p_i)
    const double *ring;
    __device__ double operator()(int arr, int q) const { return ring[arr * 3 * kRP + q]; }
};

// The predictor (ops::Pred1 then ops::Pred2) in one kernel.  A block owns
// (W-1) x (R-1) nodes of a y-z plane (k fastest) and a chunk of planes along
// x, and marches along x: for each plane i it computes Pred1 for the cells of
// plane i+1 that its nodes read (its W x R cells: the +1 halo in y and z is
// recomputed by the neighbouring block too) into a ring of three planes in
// shared memory, then Pred2 for its nodes of plane i from the ring.  cv1 and
// the half-step B never go to global memory.  The half-step p_e and p_i of
// the block's own cells go to pe_out / pi_out: in resistive runs Pred1 reads
// the step-start p_e / p_i at cells that other blocks own, so those arrays
// cannot be overwritten in place.
template <bool GEO, bool P2, int CW = 0>
__device__ __forceinline__ void pred(const Ctx &c, const MarchTile &m, int b, int resistive, double *pe_out,
                                     double *pi_out, double *ring)
{
    using P1 = ops::Pred1;  // ring: [PredRingSrc::NR][3 planes][kRP]
    const Geom &g = c.g;
    const MarchAt a = march_at<CW>(m, b, (int)threadIdx.x);
    const int W = CW ? CW : m.W;
    const int i0 = a.i0, i1 = min(i0 + m.MI - 1, g.nx);
    const int t = (int)threadIdx.x, j = a.j0 + a.pj, k = a.k0 + a.pk;
    const bool on = a.own && j <= g.ny && k <= g.nz;
    const bool cell = a.cell && j <= g.ny + 1 && k <= g.nz + 1;
    // Pred1 at the block's cells of plane i (cells 0..n+1: what Pred2 reads)
    auto produce = [&](int i) {
        if (!cell) return;
        const int slot = i % 3;
        double out[P1::NOUT];
        P1::compute<GEO, P2>(c, resistive, i, j, k, out);
#pragma unroll
        for (int q = 0; q < P1::PE; ++q) ring[(q * 3 + slot) * kRP + t] = out[q];
        ring[(P1::PE * 3 + slot) * kRP + t] = out[P1::PE] + out[P1::PI];
        if (on && i <= i1) {
            const int o = box_off(g, i, j, k);
            pe_out[o] = out[P1::PE];
            pi_out[o] = out[P1::PI];
        }
    };
    const PredRingSrc src{ring};
    produce(i0);
    for (int i = i0; i <= i1; ++i) {
        if (g.far && cell && i < i1) {
            const int o = box_off(g, i + 2, j, k);
            prefetch(c.f[SAMS_F_VX], o);
            prefetch(c.f[SAMS_F_VY], o);
            prefetch(c.f[SAMS_F_VZ], o);
            prefetch(c.f[SAMS_F_RHO], o);
            prefetch(c.f[SAMS_F_ENERGY_ELECTRON], o);
            prefetch(c.f[SAMS_F_ENERGY_ION], o);
            prefetch(c.s[S_VH], o);
            if (resistive) {
                prefetch(c.s[S_B1X], o);
                prefetch(c.s[S_B1Y], o);
                prefetch(c.s[S_B1Z], o);
                prefetch(c.s[S_PE], o);
                prefetch(c.s[S_PI], o);
            } else {
                prefetch(c.f[SAMS_F_BX], o);
                prefetch(c.f[SAMS_F_BY], o);
                prefetch(c.f[SAMS_F_BZ], o);
            }
            prefetch(c.s[S_FXV], o - g.sx);
            prefetch(c.s[S_FYV], o - g.sx);
            prefetch(c.s[S_FZV], o - g.sx);
            prefetch(c.s[S_RHOV], o - g.sx);
        }
        produce(i + 1);
        __syncthreads();  // the ring's planes i and i+1 are complete
        if (on) {
            const int s0 = i % 3, s1 = (i + 1) % 3;
            ops::Pred2::run_src<GEO, P2>(c, i, j, k, src, s0 * kRP + t, (s1 - s0) * kRP, W, 1);
        }
        // three ring planes: the next iteration's producer writes the plane
        // this one read as i-1, which no thread reads after this barrier
    }
}

// A cell op feeding a node op that reads it at the node's eight cells, in
// one kernel: the same march as pred over nodes -1..n+1 of every dimension,
// with the cell op over cells -1..n+2.  P::produce computes a cell's ring
// values (P::NR of them) and, where `own`, stores its outputs (each cell is
// owned by one block: a chunk, row or column holds its own cells and, at the
// grid's upper end, the +1 halo cell too); P::consume runs the node op from
// the ring.
template <class P, bool GEO, bool P2, int CW = 0>
__device__ __forceinline__ void cellnode(const Ctx &c, const MarchTile &m, int b, int arg, double *ring)
{
    const Geom &g = c.g;  // ring: [P::NR][3 planes][kRP]
    const MarchAt a = march_at<CW>(m, b, (int)threadIdx.x);
    const int W = CW ? CW : m.W;
    const int i0 = -1 + a.i0, i1 = min(i0 + m.MI - 1, g.nx + 1);
    const int t = (int)threadIdx.x, j = -1 + a.j0 + a.pj, k = -1 + a.k0 + a.pk;
    const bool on = a.own && j <= g.ny + 1 && k <= g.nz + 1;
    const bool cell = a.cell && j <= g.ny + 2 && k <= g.nz + 2;
    const int R = CW ? kMThreads / (CW ? CW : 1) : m.R;
    const bool own_jk = (a.pj < R - 1 || j == g.ny + 2) && (a.pk < W - 1 || k == g.nz + 2);
    auto produce = [&](int i) {
        if (!cell) return;
        const int slot = (i + 3) % 3;
        double out[P::NR];
        P::template produce<GEO, P2>(c, arg, i, j, k, own_jk && (i <= i1 || i == g.nx + 2), out);
#pragma unroll
        for (int q = 0; q < P::NR; ++q) ring[(q * 3 + slot) * kRP + t] = out[q];
    };
    const RingSrc src{ring};
    produce(i0);
    for (int i = i0; i <= i1; ++i) {
        if (g.far && cell && i < i1) P::prefetch_cell(c, box_off(g, i + 2, j, k));
        produce(i + 1);
        __syncthreads();  // the ring's planes i and i+1 are complete
        if (on) {
            const int s0 = (i + 3) % 3, s1 = (i + 4) % 3;
            P::template consume<GEO, P2>(c, arg, i, j, k, src, s0 * kRP + t, (s1 - s0) * kRP, W, 1);
        }
    }
}

// CellPrep + NodePrep: each cell's rho and sound speed go into the ring for
// the node averages, so cs never goes to global memory; in resistive runs
// (arg 1) the cell's step-start p_e, p_i are stored.
struct PrepMarch {
    __device__ static void prefetch_cell(const Ctx &c, int o)
    {
        prefetch(c.f[SAMS_F_RHO], o);
        prefetch(c.f[SAMS_F_ENERGY_ELECTRON], o);
        prefetch(c.f[SAMS_F_ENERGY_ION], o);
        prefetch(c.f[SAMS_F_BX], o);
        prefetch(c.f[SAMS_F_BY], o);
        prefetch(c.f[SAMS_F_BZ], o);
    }
    static constexpr int NR = 2, kMinBlocks = 4;  // register cap tuned on B200
    template <bool GEO, bool P2>
    __device__ static void produce(const Ctx &c, int resistive, int i, int j, int k, bool own, double *out)
    {
        const int o = box_off(c.g, i, j, k);
        double pe, pi;
        out[1] = ops::CellPrep::sound_speed(c, o, out[0], pe, pi);
        if (resistive && own) {
            c.s[S_PE][o] = pe;
            c.s[S_PI][o] = pi;
        }
    }
    template <bool GEO, bool P2, class S>
    __device__ static void consume(const Ctx &c, int, int i, int j, int k, const S &src, int q0, int QX, int QY, int QZ)
    {
        ops::NodePrep::run_src<GEO, P2>(c, i, j, k, src, q0, QX, QY, QZ);
    }
};

// SweepVol + SweepCvc of one sweep: cv1 goes into the ring for the node
// volumes cvc1.
template <int DIR>
struct VolMarch {
    __device__ static void prefetch_cell(const Ctx &c, int o)
    {
        if (DIR == 0) prefetch(c.f[SAMS_F_VX1], o);
        if (DIR <= 1) prefetch(c.f[SAMS_F_VY1], o);
        prefetch(c.f[SAMS_F_VZ1], o);
    }
    static constexpr int NR = 1, kMinBlocks = DIR == 2 ? 5 : 4;  // register cap tuned on B200
    template <bool GEO, bool P2>
    __device__ static void produce(const Ctx &c, int arg, int i, int j, int k, bool own, double *out)
    {
        out[0] = ops::SweepVol<DIR>::template compute<GEO, P2>(c, arg, i, j, k, own);
    }
    template <bool GEO, bool P2, class S>
    __device__ static void consume(const Ctx &c, int, int i, int j, int k, const S &src, int q0, int QX, int QY, int QZ)
    {
        ops::SweepCvc::node(c, box_off(c.g, i, j, k), src, q0, QX, QY, QZ);
    }
};

// The shock heating (Corr1) from per-edge terms.  A cell's heating sums
// twelve products of velocity jumps (lagran.cpp:888-979), one per edge
// between the cell's corner nodes, and four cells share an edge.  Each
// product is formed once, at the node where its edge ends: the march of pred
// over cells 0..n+1; for each plane i the block forms the x, y and z edge
// terms of the nodes of plane i that its cells read (rows j0-1 .. , columns
// from k0) into a ring of three planes in shared memory, then runs the cell
// op for its cells of plane i from the ring's planes i-1 and i.
// (Corr2's energy and density update folded in here, with only its velocity
// update left as a kernel, measured slower on B200: 0.83 + 0.25 ms against
// 0.43 + 0.60.)
constexpr int kHeatMinBlocks = 4;  // register cap tuned on B200
template <bool GEO, bool P2, int CW = 0>
__device__ __forceinline__ void heat_edges(const Ctx &c, const MarchTile &m, int b, double *ring)
{
    const Geom &g = c.g;  // ring: [3 edge directions][3 planes][kRP]
    const MarchAt a = march_at<CW>(m, b, (int)threadIdx.x);
    const int W = CW ? CW : m.W;
    const int i0 = a.i0, i1 = min(i0 + m.MI - 1, g.nx + 1);
    const int t = (int)threadIdx.x, jn = a.j0 - 1 + a.pj, k = a.k0 + a.pk, j = a.j0 + a.pj;
    const bool node = a.cell && jn <= g.ny + 1 && k <= g.nz + 2;
    const bool on = a.own && j <= g.ny + 1 && k <= g.nz + 1;
    auto produce = [&](int i) {
        if (!node) return;
        const int slot = (i + 3) % 3;
        double e[3];
        ops::Corr1::node_edges(c, box_off(g, i, jn, k), e);
#pragma unroll
        for (int q = 0; q < 3; ++q) ring[(q * 3 + slot) * kRP + t] = e[q];
    };
    const RingSrc src{ring};
    produce(i0 - 1);
    for (int i = i0; i <= i1; ++i) {
        if (g.far && node && i < i1) {
            const int o = box_off(g, i + 1, jn, k);
            prefetch(c.f[SAMS_F_VX], o);
            prefetch(c.f[SAMS_F_VY], o);
            prefetch(c.f[SAMS_F_VZ], o);
            prefetch(c.f[SAMS_F_VX1], o);
            prefetch(c.f[SAMS_F_VY1], o);
            prefetch(c.f[SAMS_F_VZ1], o);
            prefetch(c.s[S_A1], o);
            prefetch(c.s[S_A2], o);
            prefetch(c.s[S_A3], o);
        }
        produce(i);
        __syncthreads();  // the ring's planes i-1 and i are complete
        if (on) {
            const int s0 = (i + 3) % 3, sm = (i + 2) % 3;
            double e[12];
            ops::Corr1::ring_edges(src, s0 * kRP + t + W, (s0 - sm) * kRP, W, e);
            c.s[S_VH][box_off(g, i, j, k)] = ops::Corr1::heating_finish<GEO, P2>(c, i, j, k, e);
        }
        // three ring planes: the next iteration's producer writes the plane
        // this one read as i-2, which no thread reads any more
    }
}

// One resistive sub-step (ops::ResistRK then ops::ResistB) in one kernel,
// out of place for B.  A block owns (W-1) x (R-1) points of a y-z plane of
// the whole box (-2..n+2) and a chunk of planes along x, and marches along x:
// ResistRK for the cells of plane i that its points read (the -1 halo in y
// and z is recomputed by the neighbouring block) goes into a ring of three
// planes in shared memory, then ResistB for its points of plane i reads the
// ring's planes i-1 and i.  ResistRK reads B at +1 neighbours that other
// blocks update, so the new B goes to nbx/nby/nbz (every box point: updated
// or copied); the electron energy is updated in place (nothing else reads
// it here).
template <bool GEO, bool P2, int CW = 0>
__device__ __forceinline__ void resist(const Ctx &c, const MarchTile &m, int b, double *nbx, double *nby, double *nbz,
                                       double *ring)
{
    using RK = ops::ResistRK;  // ring: [RK::NOUT][3 planes][kRP]
    const Geom &g = c.g;
    const MarchAt a = march_at<CW>(m, b, (int)threadIdx.x);
    const int W = CW ? CW : m.W;
    const int i0 = -2 + a.i0, i1 = min(i0 + m.MI - 1, g.nx + 2);
    const int t = (int)threadIdx.x, j = -2 + a.j0 + a.pj, k = -2 + a.k0 + a.pk;
    // the thread's ring cell is (j - 1, k - 1); ResistRK is defined on 0..n
    const bool cell = a.cell && j >= 1 && j - 1 <= g.ny && k >= 1 && k - 1 <= g.nz;
    const bool on = a.own && j <= g.ny + 2 && k <= g.nz + 2;
    auto produce = [&](int i) {
        if (!cell || i < 0 || i > g.nx) return;
        const int slot = (i + 6) % 3;
        double out[RK::NOUT];
        RK::compute<GEO, P2>(c, i, j - 1, k - 1, out);
#pragma unroll
        for (int q = 0; q < RK::NOUT; ++q) ring[(q * 3 + slot) * kRP + t] = out[q];
    };
    const RingSrc src{ring};
    produce(i0 - 1);
    for (int i = i0; i <= i1; ++i) {
        if (g.far && on && i < i1) {
            const int o = box_off(g, i + 1, j, k), ob = i < g.nx ? o + g.sx : o;  // ResistRK reads B at +1
            prefetch(c.f[SAMS_F_BX], ob);
            prefetch(c.f[SAMS_F_BY], ob);
            prefetch(c.f[SAMS_F_BZ], ob);
            prefetch(c.f[SAMS_F_RHO], o);
            prefetch(c.f[SAMS_F_ENERGY_ELECTRON], o);
        }
        produce(i);
        __syncthreads();  // the ring's planes i-1 and i are complete
        if (on) {
            const int s0 = (i + 6) % 3, sm = (i + 5) % 3;
            ops::ResistB::run_src<P2>(c, i, j, k, src, s0 * kRP + t + W + 1, (s0 - sm) * kRP, W, 1, nbx, nby, nbz);
        }
    }
}

// ---------------------------------------------------------------------------
// Window kernels
// ---------------------------------------------------------------------------

// Windows of the x and y sweeps: kWinK lanes (a warp) over the flattened
// transverse plane (third index a, then k) times up to kWinS own points along
// the sweep.  Flattening keeps every lane busy whatever the row length: a
// row of 257 values is 8.03 warps, one of 5 a sixth of one.
struct WinTile {
    int S;       // own points along the sweep per window
    int nwin;    // windows along the sweep
    int groups;  // lane groups of the transverse plane
    int blocks;
};

// nd points along the sweep, `lanes` in the transverse plane.  As few windows
// as kWinS allows (each recomputes three halo points), unless that leaves
// SMs without a block: then shorter ones, whose stages take fewer rounds of
// the block's eight rows.
inline WinTile win_tile(int nd, long long lanes, int halo, int sm_blocks)
{
    WinTile w{};
    w.groups = (int)((lanes + ops::kWinK - 1) / ops::kWinK);
    const int rows = ops::kWinThreads / ops::kWinK;
    double cost = 0.0;
    for (int n = (nd + ops::kWinS - 1) / ops::kWinS; n <= nd; ++n) {
        const int S = (nd + n - 1) / n, nw = (nd + S - 1) / S;
        const long long blocks = (long long)nw * w.groups;
        const double waves = (double)blocks / sm_blocks;
        const long long whole = (blocks + sm_blocks - 1) / sm_blocks;
        const double t = (waves < 4.0 ? (double)whole : waves + 0.5) * (double)((S + halo + rows - 1) / rows + (S + rows - 1) / rows);
        if (w.S == 0 || t < cost) {
            w.S = S;
            w.nwin = nw;
            w.blocks = (int)blocks;
            cost = t;
        }
        if (waves >= 4.0) break;  // enough blocks: fewest windows
    }
    return w;
}

// Thread t of block b: own points s0..s1 along the sweep (the block's rows sl,
// sl + 8, ...), lane kc and its transverse point (a, k), k over nk values from
// 0 (a past its range: an idle lane).
struct WinAt {
    int s0, s1, sl, kc, a, k;
};
__host__ __device__ __forceinline__ WinAt win_at(const WinTile &w, int b, int t, int nd, int nk)
{
    WinAt r;
    const int win = b % w.nwin, grp = b / w.nwin;
    r.s0 = win * w.S;
    r.s1 = r.s0 + w.S - 1 < nd ? r.s0 + w.S - 1 : nd;
    r.kc = t % ops::kWinK;
    r.sl = t / ops::kWinK;
    const int q = grp * ops::kWinK + r.kc;
    r.a = q / nk;
    r.k = q - r.a * nk;
    return r;
}

// CT window store: kCtP points along the sweep (own points and the quotient
// halo of one before and two after) x kWinK lanes.
constexpr int kCtP = ops::kWinS + 3;
struct CtStore {
    double *sm;
    int at, kc;
    __device__ double get(int a, int ds) const { return sm[(a * kCtP + at + ds) * ops::kWinK + kc]; }
    __device__ void put(int a, double v) const { sm[(a * kCtP + at) * ops::kWinK + kc] = v; }
};

// SweepCT + SweepMass of the x or y sweep (ops::SweepCTMass<DIR>) over
// windows; the transverse plane is (a, k) in 0..na+1 x 0..nz+1 (a: j for x, i
// for y).  The CT quotients of the window's points and of a halo of one
// before and two after go to shared memory first.  CT fluxes where a and k
// are in 0..n, mass fluxes everywhere.
template <int DIR, bool GEO>
__device__ __forceinline__ void ctmass(const Ctx &c, const WinTile &w, int b, int scale, int images, double *csm)
{
    using F = ops::SweepCTMass<DIR>;
    constexpr int TS = ops::kWinThreads / ops::kWinK;
    const Geom &g = c.g;
    const int nd = DIR == 0 ? g.nx : g.ny, na = DIR == 0 ? g.ny : g.nx;
    const WinAt p = win_at(w, b, (int)threadIdx.x, nd, g.nz + 2);
    const int s0 = p.s0, s1 = p.s1, kc = p.kc, sl = p.sl, a = p.a, k = p.k;
    const bool mass = a <= na + 1, ct = a <= na && k <= g.nz;
    auto at = [&](int s) { return CtStore{csm, s - s0 + 1, kc}; };
    if (g.far && mass)
        for (int s = s0 + sl; s <= s1; s += TS) {
            const int o = box_off(g, DIR == 0 ? s : a, DIR == 0 ? a : s, k);
            prefetch(c.f[SAMS_F_VX1 + DIR], o);
            prefetch(c.s[S_R_CV1], o);
            prefetch(c.s[S_R_CVC1], o);
            prefetch(c.f[SAMS_F_RHO], o);
        }
    if (ct)
        for (int s = s0 - 1 + sl; s <= s1 + 2; s += TS)
            F::template quot<GEO>(c, DIR == 0 ? s : a, DIR == 0 ? a : s, k, at(s), scale != 0);
    __syncthreads();
    if (mass)
        for (int s = s0 + sl; s <= s1; s += TS)
            F::template fluxes<GEO>(c, DIR == 0 ? s : a, DIR == 0 ? a : s, k, at(s), ct, images);
}

// SweepCT + SweepMass of the z sweep: a block holds L stretches of z lines
// (i, j) in 0..nx+1 x 0..ny+1 (CT fluxes on the lines in 0..n), each of up to
// S own points and the quotient halo of one before and two after, one thread
// per point.
struct ZTile {
    int S, nseg;  // own points of a stretch, stretches per line
    int L;        // stretches per block
    int blocks;
};
constexpr int kZCtThreads = 288;
// The number of stretches per line that keeps most of the block's threads on
// own points.
inline ZTile z_tile(int nz, long long lines)
{
    ZTile z{};
    double eff = 0.0;
    for (int n = 1; n <= nz + 1; ++n) {
        const int S = (nz + n) / n, L = kZCtThreads / (S + 3);
        if (L < 1) continue;
        const int nseg = (nz + S) / S;
        const double e = (double)L * (nz + 1) / nseg / kZCtThreads;
        if (z.S == 0 || e > eff) {
            z.S = S;
            z.nseg = nseg;
            z.L = L;
            eff = e;
        }
        if (S <= 16) break;
    }
    z.blocks = (int)((lines * z.nseg + z.L - 1) / z.L);
    return z;
}
struct ZRowStore {
    double *sm;
    int at;
    __device__ double get(int a, int ds) const { return sm[a * kZCtThreads + at + ds]; }
    __device__ void put(int a, double v) const { sm[a * kZCtThreads + at] = v; }
};

// Thread t of block b: the point (i, j, k) of its line (i past nx+1 or
// !on: idle), `own` where it is one of the stretch's own points 0..nz.
struct ZAt {
    int i, j, k;
    bool on, own;
};
__host__ __device__ __forceinline__ ZAt z_at(const ZTile &z, int b, int t, const Geom &g)
{
    ZAt p;
    const int span = z.S + 3, r = t / span, kk = t - r * span;
    const long long st = (long long)b * z.L + r;
    const int line = (int)(st / z.nseg), seg = (int)(st - (long long)line * z.nseg);
    p.i = line / (g.ny + 2);
    p.j = line - p.i * (g.ny + 2);
    p.k = seg * z.S - 1 + kk;
    p.on = r < z.L && p.i <= g.nx + 1;
    p.own = p.on && kk >= 1 && kk <= z.S && p.k <= g.nz;
    return p;
}

template <bool GEO>
__device__ __forceinline__ void ctmass_z(const Ctx &c, const ZTile &z, int b, int images, double *zsm)
{
    using F = ops::SweepCTMass<2>;
    const Geom &g = c.g;
    const int t = (int)threadIdx.x;
    const ZAt p = z_at(z, b, t, g);
    const bool ct = p.on && p.i <= g.nx && p.j <= g.ny;
    if (ct && p.k <= g.nz + 2) F::quot<GEO>(c, p.i, p.j, p.k, ZRowStore{zsm, t}, false);
    __syncthreads();
    if (p.own) F::fluxes<GEO>(c, p.i, p.j, p.k, ZRowStore{zsm, t}, ct, images);
}

// The x or y sweep's stages (ops::SweepFused<DIR>) out of place, over windows;
// the transverse plane is (a, k) in 0..na x 0..nz.  The solve's state arrays
// are only read; the new rho, energies and velocities go to w.  Halo points
// recompute stage A (two before, one after) and stage B (one before) without
// writing the state.  Each own point (0..n in every dimension) also takes the
// sweep's CT update of B (SweepCTUpd<DIR> with ct_arg); no stage reads B.
template <int DIR, bool GEO>
__device__ __forceinline__ void psweep(const Ctx &c, const WinTile &wt, int b, const ops::SweepOut &w, int ct_arg,
                                       double *psm)
{
    using F = ops::SweepFused<DIR>;
    constexpr int TS = ops::kWinThreads / ops::kWinK;
    const Geom &g = c.g;
    const int nd = DIR == 0 ? g.nx : g.ny, na = DIR == 0 ? g.ny : g.nx;
    const WinAt p = win_at(wt, b, (int)threadIdx.x, nd, g.nz + 1);
    const int s0 = p.s0, s1 = p.s1, kc = p.kc, sl = p.sl, a = p.a, k = p.k;
    const bool on = a <= na;
    auto at = [&](int s) { return ops::WinStore{psm, s - s0 + 2, kc}; };
    const int a_lo = max(s0 - 2, -2), a_hi = min(s1 + 1, nd + 1);
    if (g.far && on) {
        for (int s = a_lo + sl; s <= a_hi; s += TS) {
            const int o = box_off(g, DIR == 0 ? s : a, DIR == 0 ? a : s, k);
            prefetch(c.f[SAMS_F_ENERGY_ELECTRON], o);
            prefetch(c.f[SAMS_F_ENERGY_ION], o);
            prefetch(c.s[S_R_CV1], o);
            prefetch(c.s[S_R_CVC1], o);
            prefetch(c.s[S_R_RHO1], o);
            prefetch(c.f[SAMS_F_DM], o);
            prefetch(c.f[SAMS_F_VX1 + DIR], o);
            prefetch(c.s[S_R_CV2], o);
            prefetch(c.f[SAMS_F_VX], o);
            prefetch(c.f[SAMS_F_VY], o);
            prefetch(c.f[SAMS_F_VZ], o);
        }
    }
    for (int s = a_lo + sl; s <= a_hi; s += TS)
        if (on) F::template stage_a<GEO>(c, DIR == 0 ? s : a, DIR == 0 ? a : s, k, at(s), w, s >= s0 && s <= s1);
    __syncthreads();
    for (int s = s0 + sl; s <= s1; s += TS)
        if (on) F::stage_b_energy(c, DIR == 0 ? s : a, DIR == 0 ? a : s, k, at(s), w);
    __syncthreads();
    const int b_lo = max(s0 - 1, -1);
    for (int s = b_lo + sl; s <= s1; s += TS)
        if (on) F::template stage_b_mom<GEO>(c, DIR == 0 ? s : a, DIR == 0 ? a : s, k, at(s));
    __syncthreads();
    for (int s = s0 + sl; s <= s1; s += TS)
        if (on) F::stage_c(c, DIR == 0 ? s : a, DIR == 0 ? a : s, k, at(s), w);
    for (int s = s0 + sl; s <= s1; s += TS)
        if (on) ops::SweepCTUpd<DIR>::template run<GEO, false>(c, ct_arg, DIR == 0 ? s : a, DIR == 0 ? a : s, k);
}

// The z sweep's stages S6, S7 and S8 (ops::SweepFused<2>) over whole z
// lines, in place: a block holds kZThreads / (nz + 4) lines of (i, j) in
// 0..nx x 0..ny, one thread per k = -2..nz+1 of each.  Each point of 0..n also
// takes the z sweep's CT update of B (SweepCTUpd<2> with ct_arg), which
// nothing else in the kernel reads or writes.
constexpr int kZThreads = ops::kZLineThreads;
template <bool GEO>
__device__ __forceinline__ void zsweep(const Ctx &c, int b, int ct_arg, double *zsm)
{
    using F = ops::SweepFused<2>;
    static_assert(!F::kSharedFluxSlots, "the z passes of stage B run without a barrier between them");
    static_assert(std::is_same<typename F::EnergyIn, const double *>::value, "arrays written in place are not read as RO");
    const Geom &g = c.g;
    const int W = g.nz + 4, lines = kZThreads / W, S = lines * W;
    const int line = (int)threadIdx.x / W, k = (int)threadIdx.x % W - 2;
    const long long q = (long long)b * lines + line;
    const bool on = line < lines && q < (long long)(g.nx + 1) * (g.ny + 1);
    const int i = on ? (int)(q / (g.ny + 1)) : 0, j = on ? (int)(q % (g.ny + 1)) : 0;
    const ops::LineStore st{zsm, S, line * W + k + 2};
    const ops::SweepOut w = ops::sweep_in_place(c);
    if (g.far && on) {
        const int o = box_off(g, i, j, k);
        prefetch(c.f[SAMS_F_VX], o);
        prefetch(c.f[SAMS_F_VY], o);
        prefetch(c.f[SAMS_F_VZ], o);
        prefetch(c.s[S_R_CV2], o);
        prefetch(c.f[SAMS_F_DM], o);
        prefetch(c.f[SAMS_F_ENERGY_ELECTRON], o);
        prefetch(c.f[SAMS_F_ENERGY_ION], o);
        prefetch(c.f[SAMS_F_BX], o);
        prefetch(c.f[SAMS_F_BY], o);
        prefetch(c.f[SAMS_F_BZ], o);
        prefetch(c.s[S_R_CT1], o);
        prefetch(c.s[S_R_CT2], o);
    }
    if (on) F::stage_a<GEO>(c, i, j, k, st, w, true);
    __syncthreads();
    if (on && k >= 1 && k <= g.nz) F::stage_b_energy(c, i, j, k, st, w);
    if (on && k >= -1 && k <= g.nz) F::stage_b_mom<GEO>(c, i, j, k, st);  // its own slots: no barrier between
    __syncthreads();
    if (on && k >= 0 && k <= g.nz) F::stage_c(c, i, j, k, st, w);
    if (on && k >= 0 && k <= g.nz) ops::SweepCTUpd<2>::run<GEO, false>(c, ct_arg, i, j, k);
}

}  // namespace march
}  // namespace sams
