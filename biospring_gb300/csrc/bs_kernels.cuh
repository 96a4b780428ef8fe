// bs_kernels.cuh -- kernel declarations of the GB300 step engine.
#pragma once

#include "bs_common.cuh"

namespace bsg
{

constexpr int kStepBlock = 128; // adjoint and diagnostic kernels
#ifndef BS_STEP_BLOCK
#define BS_STEP_BLOCK 256
#endif
#ifndef BS_STEP_MIN_BLOCKS
#define BS_STEP_MIN_BLOCKS (1024 / BS_STEP_BLOCK)
#endif
// threads per block of the step kernel, and the resident blocks per SM it is compiled for
// (1024 resident threads: at most 64 registers)
constexpr int kStepKernelBlock = BS_STEP_BLOCK;
constexpr int kStepMinBlocks = BS_STEP_MIN_BLOCKS;
constexpr int kStepPartBlock = 128; // of the steps whose energies are not summed
constexpr int kBuildLanes = 8;    // threads per slot of the spring-table rebuild when the table fits L2
// k_order: most blocks of its grid, and the threads a particle it is sized for (small systems use as few
// blocks as their spring table needs, for cheaper barriers)
constexpr int kOrderMaxBlocks = 1024;
constexpr int kOrderLanes = 8;

// status bits that stop a rebuild; a stale list is what a rebuild repairs
constexpr int kRebuildBlocking = ST_NONFINITE | ST_PAIR_CAPACITY | ST_CELL_CAPACITY | ST_WIDE | ST_BARRIER;
// Coulomb rows walked by the whole warp, one charged particle at a time, instead of by the
// particle's own lanes (100k step after an L2 flush: 112.0 -> 110.8 us; warm: unchanged).
#ifndef BS_COUL_WARP
#define BS_COUL_WARP 1
#endif
// Programmatic dependent launch: the list builds begin launching while k_order runs. Step kernels keep full
// stream ordering: launched early they take the slots of the step before them (calls of 20 steps at
// 100,000 particles 1,557 -> 1,768 us with the trigger at their start, 1,591 us with it at their end).
#ifndef BS_PDL
#define BS_PDL 1
#endif
// Gathers in flight per lane in the step kernel's spring and steric loops: kGatherU entries are
// read per pass and their partners loaded together (0: the entry-by-entry software-pipelined
// loops). BS_GATHER_BATCH selects it for the persistent ensemble kernel (512 Calpha networks of
// degree 19: 2.19e9 -> 2.96e9 particle-steps/s); both forms sum the same entries in the same order.
#ifndef BS_GATHER
#define BS_GATHER 3
#endif
#ifndef BS_GATHER_BATCH
#define BS_GATHER_BATCH 1
#endif
constexpr int kGatherU = 4;
// the LJ pair body refines the hardware reciprocal by one Newton step (0: the approximation alone)
#ifndef BS_LJ_RCP_REFINE
#define BS_LJ_RCP_REFINE 1
#endif
#ifndef BS_LJ_BAND_AFTER
#define BS_LJ_BAND_AFTER 0
#endif
#ifndef BS_HOIST
#define BS_HOIST 1
#endif
// the lean step kernel (BS_LEAN 0: always the full one)
#ifndef BS_LEAN
#define BS_LEAN 1
#endif
// Dense list build: cells of half the list radius, in groups of 2 x 2 x 2 cells per block (bs_list.cu).
#ifndef BS_GRID_DIV
#define BS_GRID_DIV 2
#endif
constexpr int kGridDiv = BS_GRID_DIV; // cell-block list build: cells per list radius (stencil of +-kGridDiv cells)
constexpr int kSparseDiv = 1;         // warp-per-particle list build (sparse systems, batches): cells of the radius

enum StepMode
{
    MODE_STEP = 0,   // forces + Euler step (SpringNetwork::computeStep)
    MODE_FORCES = 1, // forces and energies only (SpringNetwork::computeForces)
    // A step with further steps enqueued behind it in the same call: every way to read energies completes
    // those first (or fails), so this step's could not be seen and are not summed.
    MODE_STEP_PART = 2,
};

// Launchers (all asynchronous on `stream`); each returns the number of kernels launched.
int launch_rebuild(const Params &p, cudaStream_t stream);
cudaError_t launch_order(const Params &p, cudaStream_t stream); // bs_order.cu
cudaError_t order_blocks(const Params &p, int *blocks);
size_t order_bins(const Params &p); // entries of Params::cell_bin (single systems)
int launch_pairlist(const Params &p, cudaStream_t stream); // bs_list.cu
int launch_step(const Params &p, int mode, cudaStream_t stream);      // step kernel, then the bodies
int launch_step_only(const Params &p, int mode, cudaStream_t stream); // the step kernel alone
int launch_rigid(const Params &p, cudaStream_t stream);               // bs_rigid.cu
// count steps without a rebuild in between: one kernel where the system allows (Params::run_on)
int launch_steps(const Params &p, int count, cudaStream_t stream);
// bs_run.cu: the kernel of several steps, its blocks, and whether they are resident at once
// (save, save_lo, nullable: the positions every step starts from and their remainders, npad a step)
cudaError_t launch_run(const Params &p, int count, cudaStream_t stream, float4 *save = nullptr,
                       float4 *save_lo = nullptr);
cudaError_t run_fits(Params &p); // sets run_on and run_hold
int run_blocks(const Params &p);
// the kernel for a steric form (null where there is none for these lanes and this hold)
const void *run_linear(int lanes, bool lean, int hold);
const void *run_amber(int lanes, bool lean, int hold);
const void *run_lewitt(int lanes, bool lean, int hold);
const void *run_zacharias(int lanes, bool lean, int hold);
// Steps of one launch (10 in the default schedule) and the polls after which a barrier gives up (Params::
// barrier_polls; some seconds, a meeting takes about a microsecond).
constexpr int kRunMaxSteps = 1024;
constexpr int kBarrierPolls = 1 << 22;
// The lean step kernels leave out, at compile time, the terms most systems do not use (pairwise
// hydrophobic forces, field grids, the probe, rigid bodies, float-float positions): fewer live
// registers, so the common kernel runs without register spills.
inline bool lean_step(const Params &p)
{
    return BS_LEAN && !(p.hydro_on || p.fg_on[0] || p.fg_on[1] || p.probe_on || p.nbody > 0 || p.pos_lo[0]);
}
int launch_ext_add(const Params &p, long long i, float fx, float fy, float fz, cudaStream_t stream);
int launch_set_burying(const Params &p, const float *burying, cudaStream_t stream);
int launch_set_charges(const Params &p, const float *q, cudaStream_t st);
// new stiffness and rest length (nullable, by spring) into the nnz entries of the caller-order spring table
int launch_set_springs(const Params &p, int nnz, const unsigned int *sid, const float *k, const float *r0, cudaStream_t st);
// Loads the module of the step and state kernels (9 ms, once a process), which is otherwise loaded by the first
// launch of one of them: a getter, for a small system. Called at set-up.
cudaError_t load_step_kernels();
int launch_unsort(const Params &p, int what, float *out3, cudaStream_t stream);
int launch_diag_cells(const Params &p, float cutoff, float skin, uint32_t need_flag, long long *out,
                      cudaStream_t stream);
int launch_diag_pairs(const Params &p, int term, long long *out, unsigned long long *count,
                      unsigned long long cap, cudaStream_t stream);
int launch_set_positions(const Params &p, const float *xyz, const float *vel, cudaStream_t stream,
                         const float *lo = nullptr);

// Discrete adjoint (bs_adjoint.cu).
struct AdjState
{
    const float4 *x;   // positions at the start of the step being reversed (sorted layout)
    const float4 *xlo; // their rounding remainders (precise_positions), else null
    float4 *lx;      // dL/dx
    float4 *lv;      // dL/dv
    float4 *nu_in;   // b (lambda_v + dt lambda_x) of the later step
    float4 *nu_out;  // the same for the step being reversed
    float *gk;       // per directed spring entry: dL/dk, dL/dr0 partial sums
    float *gr0;
    float *gq;       // dL/dq per caller id (null: no charge gradients)
};
int launch_adj_step(const Params &p, const AdjState &a, cudaStream_t stream);
// count backward steps in one kernel with `lanes` lanes a particle, the most (of 16, 8, 4) whose grid is
// resident at once (0: none is)
cudaError_t adj_run_lanes(const Params &p, int *lanes);
cudaError_t launch_adj_run(const Params &p, const AdjState &a, int count, int lanes, cudaStream_t stream);
int launch_adj_init(const Params &p, const AdjState &a, const float *target, double *blk, unsigned int *done,
                    double *loss, cudaStream_t stream);
int launch_adj_permute(const Params &p, const AdjState &a, float4 *cx, float4 *cv, int dir, cudaStream_t stream);
int launch_adj_save(const Params &p, float4 *dst, float4 *dst_lo, cudaStream_t stream);
int launch_adj_combine(int nsp, const float *gk, const float *gr0, float *ok, float *or0, cudaStream_t stream);

// Batched ensembles (bs_batch.cu).
constexpr int kBatchMaxBlock = 512; // largest block of the persistent step kernel
struct BatchShape
{
    int block;   // threads per block
    int lanes;   // threads per particle (1, 2, 4, 8)
    int cluster; // mean blocks per group (1, 2, 4, 8)
};
int launch_batch_pairlist(const Params &p, cudaStream_t stream);
cudaError_t launch_batch_run(const Params &p, const BatchShape &shape, int chunk, cudaStream_t stream);
int launch_batch_finish(const Params &p, int chunk, cudaStream_t stream);
cudaError_t batch_max_blocks(const Params &p, const BatchShape &shape, int *out); // resident at once
constexpr int kBatchMaxBlocks = 4096; // of a launch
constexpr int kBatchCatchUp = 65536;  // steps of one system in a launch, or the launch's own if those are more

} // namespace bsg
