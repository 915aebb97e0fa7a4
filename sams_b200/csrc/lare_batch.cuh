// lare_batch.cuh -- many independent LARE3D solves stepped together.
//
// Every phase of the step is ONE persistent launch over a worklist drawn from
// all live solves: the blocks of each solve's own tiling (the fused phases), or
// tiles of one solve, a slab of tile_i planes along x and a chunk of 256 points
// of the (y, z) plane (the per-point phases).  Each solve keeps its
// own state, scratch, metrics and device scalars, so each advances with its
// own CFL timestep; the batch shares only the launches.  The whole batched
// step is recorded once into a CUDA graph and replayed until the set of
// solves or the tiling changes.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <string>
#include <vector>

#include "lare_device.cuh"
#include "lare_march.cuh"
#include "lare_solver.cuh"
#include "sams_lare.h"

namespace sams {

struct Tile {
    int inst;  // slot of the solve in the batch's Ctx table
    int i0;    // first x plane of the slab
    int p0;    // first flattened (y, z) point of the chunk
    int pad;
};

// One block of a fused phase: of which solve, and which of its blocks.
struct BlockRef {
    int inst, block;
};

// One solve's tilings of the fused phases and how its ghosts are filled.
struct SolveTiles {
    march::MarchTile cellnode, pred, heat, resist;
    march::WinTile ct[2], stage[2];
    march::ZTile ctz;
    int images[3];              // what the CT + mass kernels write of dm's ghosts, per sweep
    int refilled, b_refilled;   // a fill rewrites every ghost of rho, energies and velocities; of B
    unsigned periodic, compose; // fields that the one-pass fills take (bit per field)
};

struct BatchSlot {
    bool live = false;
    sams_lare_params p{};
    BcTable bc{};
    Ctx ctx{};
    double *arena = nullptr;
    double *axes = nullptr;
    Scalars *sc = nullptr;
    long long bytes = 0;
};

class Batch {
public:
    Batch() = default;
    ~Batch();
    Batch(const Batch &) = delete;
    Batch &operator=(const Batch &) = delete;

    int init(int device);
    int set_stream(cudaStream_t s);
    int add(const sams_lare_params &p, const sams_lare_bcs &bcs, int *id);
    int remove(int id);
    int upload(int id, int field, const double *src, cudaMemcpyKind kind);
    int download(int id, int field, double *dst, cudaMemcpyKind kind);
    int download_async(int id, int field, double *dst);
    int step(long long nsteps);
    int step_graph(long long nsteps);
    int sync();
    int scalars(int id, Scalars &out);
    int set_tuning(int tile_i, int blocks_per_sm);
    int autotune(int trial_steps, int *tile_i, int *blocks_per_sm, double *best_ms);
    long long device_bytes() const;
    int live_count() const;
    long long live_cells() const;
    static long long bytes_for(const sams_lare_params &p);
    cudaStream_t stream() const { return stream_; }

    std::string err;

    // Contexts of a solve through a step (the out-of-place phases trade
    // arrays): at its start, after the first resistive sub-step, after the
    // last, from the corrector on, and in the x and y sweeps.
    enum { C_START, C_SUB, C_PRED, C_REMAP, C_X, C_Y, NCTX };

private:
    int check(cudaError_t e, const char *what);
    int rebuild();
    void enqueue_step();
    template <class Op> void launch(int ctx, int arg);
    void launch_visc();
    template <class P> void launch_cellnode(int ctx, int arg);
    void launch_resist(int ctx);
    void launch_pred(int ctx);
    void launch_heat(int ctx);
    template <int DIR> void launch_ctmass(int ctx, int scale);
    template <int DIR> void launch_psweep(int ctx, int ct_arg);
    void launch_zsweep(int ctx, int ct_arg);
    template <int DIR> void stages(int ctx, int ct_arg);
    void bc_fill(int ctx, unsigned mask, bool resistive_only);
    void bc_edges(int ctx, unsigned mask, int d, bool dm_only, bool resistive_only);
    void drop_graphs();
    void free_slot(BatchSlot &s);
    unsigned repack_grid(const Geom &g) const;

    int device_ = 0;
    cudaStream_t own_stream_ = nullptr;
    cudaStream_t stream_ = nullptr;
    std::vector<BatchSlot> slots_;
    bool dirty_ = true;
    int tile_i_ = 2;
    int blocks_per_sm_ = 4;
    int sm_count_ = 148;
    // device tables, one buffer (rebuilt when the set of solves changes)
    char *d_tables_ = nullptr;
    Ctx *d_ctx_[NCTX] = {};
    Tile *d_tiles_ = nullptr;  // plane tiles of the per-point phases
    int ntiles_ = 0;
    SolveTiles *d_st_ = nullptr;
    enum { P_CELLNODE, P_RESIST, P_PRED, P_HEAT, P_CTX, P_CTY, P_CTZ, P_STX, P_STY, P_STZ, P_FILL, NPHASE };
    BlockRef *d_list_[NPHASE] = {};  // blocks of the fused phases
    int nlist_[NPHASE] = {};
    bool fused_xy_ = false;  // the x and y sweeps' S6-S8 run as one kernel (no live solve uses rke)
    bool zfuse_ = false;     // ... the z sweep's (and every z line fits a block)
    bool fold_ = false;      // B's scaling is folded into the x and z sweeps' CT updates
    int shell_ = 0;          // some solve's ghosts outlive a fill: the out-of-place sweeps copy them
    int edges_ = 0;          // some solve has conditions that no one-pass fill takes
    bool dm_edges_[3] = {};  // some solve's dm is filled by kb_bc_edge along this dimension
    int *d_live_ = nullptr;
    BcTable *d_bc_ = nullptr;           // per slot boundary conditions
    long long *d_slab_off_ = nullptr;   // 3 x prefix of one-edge slab points per live solve
    long long slab_total_[3] = {0, 0, 0};
    int nlive_ = 0;
    int has_resistive_ = 0;
    int has_rke_ = 0;
    int has_geo_ = 0;
    int all_pow2_ = 0;  // every live solve has a power-of-two grid
    size_t table_cap_bytes_ = 0;
    std::map<long long, cudaGraphExec_t> graphs_;
};

}  // namespace sams
