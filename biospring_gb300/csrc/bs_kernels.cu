// bs_kernels.cu -- sm_103a kernels of BioSpring's per-step force-and-integrate loop.
//
// Data layout (all in HBM, structure of arrays, particles in cell-sorted order):
//   pos[2]    float4 (x, y, z, P)   double-buffered: a step reads one and writes the other
//   vel[2]    float4 (vx, vy, vz, 0)
//   fhi/chg/hyd/flags/iprm[2]       per-particle parameters, re-laid out at every rebuild
//   perm[2]   sorted slot -> caller id;  inv: caller id -> sorted slot
//   se_*      springs of each slot, ELL column-major [k * npad + slot] (coalesced per warp),
//             rows ascending by partner slot
//   pl[t]     typed nonbonded pair lists (steric dynamic / static partners, Coulomb,
//             hydrophobic), row-major [slot * cap + k], entries ascending, rebuilt every K steps
//             from the cell grid; the steric row holds 16-bit slot offsets when they fit
//
// Steric factors: the pair parameters of the LJ forms factor per particle,
// eps_ij r_ij^m = (a_i b_i^m)(a_j b_j^m) with eps_ij = a_i a_j and r_ij = b_i b_j
// (Amber/Lewitt: a = sqrt(eps), b = sqrt(r), CombinationRules.hpp:18-31; Zacharias: a = eps,
// b = r), so P = a b^6 and fhi = a b^12 (Amber) or a b^8 (Lewitt, Zacharias); the LJ path
// then needs only 1/r^2 (no square root, no division).
//
// Rebuild (every K steps, or when a particle drifted more than skin/2):
//   k_order (bs_order.cu) -> k_pairlist (bs_list.cu), or k_batch_pairlist or k_home_pairlist (bs_batch.cu) for sparse
//   systems
// Step: k_step, T consecutive lanes per particle, gathers its springs and nonbonded pairs (no
// atomics on forces, so results are deterministic) and integrates in the same pass; where the grid is resident at
// once k_run (bs_run.cuh) takes all steps up to the next rebuild.
//
// Reference behaviour reproduced (paths inside the BioSpring project):
//   cell grid and cell id           src/nsearch.hpp:277-293, 342-390 (FP64, same formula; the
//                                   search grid uses edge (cutoff + skin) / kGridDiv, the
//                                   diagnostic grid of bs_get_cells the reference edge)
//   pair filters                    src/nsearch.hpp:230 (FP64 distance) and src/spn/Particle.cpp:
//                                   213-224 (spring exclusion, float distance < cutoff, != 0),
//                                   :209 (static neighbour: full energy, no force on it)
//   force expressions               src/forcefield/energy/{spring,steric,electrostatic,hydrophobic,imp}.hpp
//   viscosity and Euler step        src/spn/Particle.cpp:80-84, 109-128
//   non-finite position check       src/spn/SpringNetwork.cpp:222-229 (status bit, no abort)

#include "bs_device.cuh"

namespace bsg
{

namespace
{

// Raised bits take effect for the following kernels only, so every block of a launch sees the same status
// at entry. One thread, after every block is done.
__device__ __forceinline__ void merge_pending(Ctl *ctl)
{
    const int pend = atomicExch(&ctl->status_pending, 0);
    if (pend)
        atomicOr(&ctl->status, pend);
}

__device__ __forceinline__ void complete_step(Ctl *ctl, int sb)
{
    ctl->sbuf = sb ^ 1;
    ctl->steps += 1;
    ctl->ext_pending = 0;
    merge_pending(ctl);
}

// One step (or one force evaluation) for every particle. T consecutive lanes share a particle:
// each takes every T-th entry of the particle's spring row and pair lists, the group sums its
// partial forces with shuffles, and the group's first lane adds the per-particle terms and
// integrates. T > 1 gives the latency-bound gather loops T times more independent loads in
// flight than one thread per particle would.
template <int MODE, int SM, int T, bool LEAN>
__global__ void __launch_bounds__(kStepKernelBlock, kStepMinBlocks) k_step(Params p)
{
    pdl_enter();
    Ctl *ctl = p.ctl;
    if (status_of(ctl) != 0)
        return;
    const int sb = ctl->sbuf, lb = ctl->lbuf;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    float e[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int pend = particle_step<MODE, SM, T, true, LEAN>(p, g / T, g % T, p.n, sb, lb, ctl->ext_pending != 0,
                                                               &ctl->probe_pos, e);
    if (MODE == MODE_STEP_PART)
    {
        // No energies: one counter finds the last block, which completes the step. The device-wide fences
        // are for raised bits only, what else a step writes is read by later kernels. The block and
        // device-wide sums had been 13% of a step at 100,000 particles; measured with this, calls of 20 and
        // 10 steps and their rebuilds: 100,000 particles 1,874 -> 1,728 us, 300,007 2,821 -> 2,647 us.
        const int any = __syncthreads_or(pend);
        if (pend)
            atomicOr(&ctl->status_pending, pend);
        if (any)
        {
            __threadfence();
            __syncthreads();
        }
        if (threadIdx.x == 0 && atomicAdd(&ctl->done_step, 1u) == gridDim.x - 1)
        {
            __threadfence();
            complete_step(ctl, sb);
            ctl->done_step = 0u;
        }
        return;
    }
    if (pend)
        atomicOr(&ctl->status_pending, pend);
    if (reduce_energies<6, kStepKernelBlock>(e, p.blk_energy, p.blk_cap, &ctl->done_step, ctl->energies))
    {
        if (threadIdx.x == 0)
        {
            publish_energies(ctl);
            if (MODE == MODE_STEP)
                complete_step(ctl, sb);
            else
                merge_pending(ctl);
        }
    }
}

// The probe's own step, after the step kernel (SpringNetwork.cpp:156-182): the sum of the
// particles' reactions (float-float, fixed order), viscosity from its velocity, the Euler step
// (Particle.cpp:109-128) and its kinetic energy, added to the step's total. One block.
__global__ void __launch_bounds__(1024) k_probe(Params p)
{
    pdl_enter();
    Ctl *ctl = p.ctl;
    const long long steps = *(volatile const long long *)&ctl->steps;
    if (steps == ctl->probe_steps)
        return; // the step kernel did not run
    float acc[3][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    for (int s = threadIdx.x; s < p.n; s += blockDim.x)
    {
        const float4 f = p.probe_f[s];
        ff_add(acc[0][0], acc[0][1], f.x, 0.f);
        ff_add(acc[1][0], acc[1][1], f.y, 0.f);
        ff_add(acc[2][0], acc[2][1], f.z, 0.f);
    }
    __shared__ float sh[3][2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        float hi = acc[k][0], lo = acc[k][1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            const float h2 = __shfl_down_sync(0xffffffffu, hi, o);
            const float l2 = __shfl_down_sync(0xffffffffu, lo, o);
            ff_add(hi, lo, h2, l2);
        }
        if (lane == 0)
        {
            sh[k][0][warp] = hi;
            sh[k][1][warp] = lo;
        }
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    float F[3];
    for (int k = 0; k < 3; ++k)
    {
        float hi = 0.f, lo = 0.f;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w)
            ff_add(hi, lo, sh[k][0][w], sh[k][1][w]);
        F[k] = __fadd_rn(hi, lo);
    }
    float4 v = ctl->probe_vel, x = ctl->probe_pos;
    float ke;
    probe_advance(p, F, x, v, ke);
    ctl->probe_pos = x;
    ctl->probe_vel = v;
    ctl->energies[BS_ENERGY_KINETIC] += static_cast<double>(ke);
    ctl->probe_steps = steps;
}

// ------------------------------------------------------------------------------------------
// Host-facing helpers
// ------------------------------------------------------------------------------------------

// Writes positions (what = 0), velocities (1), forces of the last force-only evaluation (2) or
// the positions' rounding remainders (3, precise_positions) in caller order as float[3n].
__global__ void k_unsort(Params p, int what, float *out)
{
    const Ctl *ctl = p.ctl;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.n)
        return;
    if (what == 2)
    {
        const float4 f = p.force_out[s];
        out[3 * s] = f.x;
        out[3 * s + 1] = f.y;
        out[3 * s + 2] = f.z;
        return;
    }
    const int id = p.perm[ctl->lbuf][s];
    float4 q;
    if (what == 3)
        q = p.pos_lo[0] ? p.pos_lo[ctl->sbuf][s] : make_float4(0.f, 0.f, 0.f, 0.f);
    else
        q = what == 0 ? p.pos[ctl->sbuf][s] : p.vel[ctl->sbuf][s];
    out[3 * id] = q.x;
    out[3 * id + 1] = q.y;
    out[3 * id + 2] = q.z;
}

// Overwrites positions and/or velocities from caller-order float[3n] arrays (nullable); new
// positions get the rounding remainders `lo` (float[3n], nullable: zero).
__global__ void k_set_state(Params p, const float *xyz, const float *vel, const float *lo)
{
    const Ctl *ctl = p.ctl;
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= p.n)
        return;
    const int s = p.inv[id];
    if (xyz)
    {
        float4 q = p.pos[ctl->sbuf][s];
        q.x = xyz[3 * id];
        q.y = xyz[3 * id + 1];
        q.z = xyz[3 * id + 2];
        p.pos[ctl->sbuf][s] = q;
        if (p.pos_lo[0])
            p.pos_lo[ctl->sbuf][s] = lo ? make_float4(lo[3 * id], lo[3 * id + 1], lo[3 * id + 2], 0.f)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (vel)
        p.vel[ctl->sbuf][s] = make_float4(vel[3 * id], vel[3 * id + 1], vel[3 * id + 2], 0.f);
}

// Reference cell id of each particle for a grid of edge (cutoff + skin) over the bounding box of
// all particles (nsearch.hpp:277-293, 342-390); -1 for particles without `need_flag`. One block.
__global__ void __launch_bounds__(1024) k_diag_cells(Params p, float cutoff, float skin, uint32_t need_flag,
                                                     long long *out)
{
    const Ctl *ctl = p.ctl;
    const float4 *pos = p.pos[ctl->sbuf];
    const unsigned int *fl = p.flags[ctl->lbuf];
    __shared__ float smin[3][32], smax[3][32];
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int i = threadIdx.x; i < p.n; i += blockDim.x)
    {
        const float4 q = pos[i];
        mn[0] = fminf(mn[0], q.x);
        mn[1] = fminf(mn[1], q.y);
        mn[2] = fminf(mn[2], q.z);
        mx[0] = fmaxf(mx[0], q.x);
        mx[1] = fmaxf(mx[1], q.y);
        mx[2] = fmaxf(mx[2], q.z);
    }
    for (int k = 0; k < 3; ++k)
        for (int o = 16; o > 0; o >>= 1)
        {
            mn[k] = fminf(mn[k], __shfl_down_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_down_sync(0xffffffffu, mx[k], o));
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < 3; ++k)
        {
            smin[k][warp] = mn[k];
            smax[k][warp] = mx[k];
        }
    __syncthreads();
    float bmn[3], bmx[3];
    for (int k = 0; k < 3; ++k)
    {
        bmn[k] = smin[k][0];
        bmx[k] = smax[k][0];
        for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w)
        {
            bmn[k] = fminf(bmn[k], smin[k][w]);
            bmx[k] = fmaxf(bmx[k], smax[k][w]);
        }
    }
    const float radius = cutoff + skin;
    int nc[3];
    for (int k = 0; k < 3; ++k)
    {
        const double len = __dsub_rn(static_cast<double>(bmx[k]), static_cast<double>(bmn[k]));
        nc[k] = static_cast<int>(ceil(__ddiv_rn(len, static_cast<double>(radius))) + 1.0);
    }
    for (int s = threadIdx.x; s < p.n; s += blockDim.x)
    {
        const int id = p.perm[ctl->lbuf][s];
        if (need_flag && !(fl[s] & need_flag))
        {
            out[id] = -1;
            continue;
        }
        const float4 q = pos[s];
        const long long cx = ref_cell_coord(q.x, static_cast<double>(bmn[0]), radius, nc[0]);
        const long long cy = ref_cell_coord(q.y, static_cast<double>(bmn[1]), radius, nc[1]);
        const long long cz = ref_cell_coord(q.z, static_cast<double>(bmn[2]), radius, nc[2]);
        out[id] = cx + cy * nc[0] + cz * static_cast<long long>(nc[0]) * nc[1];
    }
}

// Emits the unique interacting pairs of one term, using the step kernel's classification,
// as caller ids (min, max). Pairs of two dynamic particles are emitted once, from the lower id.
__global__ void __launch_bounds__(kStepBlock) k_diag_pairs(Params p, int term, long long *out,
                                                           unsigned long long *count, unsigned long long cap)
{
    const Ctl *ctl = p.ctl;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= p.n)
        return;
    const float4 *pos = p.pos[ctl->sbuf];
    const unsigned int fi = p.flags[ctl->lbuf][s];
    if (fi & PF_STATIC)
        return;
    if (!p.pl[term].on)
        return;
    const float4 pi = pos[s];
    const int idi = p.perm[ctl->lbuf][s];
    float lo2 = p.lo2_s, hi2 = p.hi2_s, cut = p.c_steric;
    if (term == BS_TERM_COULOMB)
    {
        lo2 = p.lo2_c;
        hi2 = p.hi2_c;
        cut = p.c_coulomb;
    }
    else if (term == BS_TERM_HYDROPHOBIC)
    {
        lo2 = p.lo2_h;
        hi2 = p.hi2_h;
        cut = p.c_hydro;
    }
    // the steric term has two lists: dynamic partners (0) and static partners (3)
    for (int pass = 0; pass < 2; ++pass)
    {
    const int li = pass == 0 ? term : kListStericStatic;
    if (pass == 1 && term != BS_TERM_STERIC)
        break;
    const PairList &L = p.pl[li];
    const int cnt = L.cnt[s];
    for (int k = 0; k < cnt; ++k)
    {
        unsigned int e;
        const size_t pos_in_row = static_cast<size_t>(s) * L.cap + k;
        if (li == 0 && p.pl16)
            e = static_cast<unsigned int>(s + reinterpret_cast<const short *>(L.idx)[pos_in_row]);
        else
            e = L.idx[pos_in_row];
        const int j = static_cast<int>(e & kSlotMask);
        const float4 pj = pos[j];
        const int idj = p.perm[ctl->lbuf][j];
        const bool j_static = (p.flags[ctl->lbuf][j] & PF_STATIC) != 0;
        if (!j_static && idj < idi)
            continue;
        const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (!pair_in(r2, lo2, hi2, pi, pj, cut, term != BS_TERM_STERIC))
            continue;
        const unsigned long long at = atomicAdd(count, 1ull);
        if (at < cap)
        {
            out[2 * at] = min(idi, idj);
            out[2 * at + 1] = max(idi, idj);
        }
    }
    }
}

} // namespace

template <typename... KArgs, typename... Args>
static void launch_plain(void (*kern)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                         Args &&...args)
{
    kern<<<grid, block, smem, st>>>(std::forward<Args>(args)...);
}

int launch_rebuild(const Params &p, cudaStream_t st)
{
    launch_order(p, st);
    int launched = 1;
    if (p.lists_off)
        return launched;
    if (p.nsys > 0 || p.pl_sparse)
        return launched + launch_batch_pairlist(p, st);
    return launched + launch_pairlist(p, st);
}

template <int MODE, int SM>
static void launch_step_lanes(const Params &p, cudaStream_t st, bool part)
{
    const long long threads_per = p.step_lanes;
    const int nb = static_cast<int>((static_cast<long long>(p.n) * threads_per + kStepKernelBlock - 1) / kStepKernelBlock);
    const int np = static_cast<int>((static_cast<long long>(p.n) * threads_per + kStepPartBlock - 1) / kStepPartBlock);
    const bool lean = lean_step(p);
    switch (p.step_lanes)
    {
    case 2:
        launch_plain(k_step<MODE, SM, 2, false>, nb, kStepKernelBlock, 0, st, p);
        break;
    case 8:
        if (lean)
            launch_plain(k_step<MODE, SM, 8, true>, nb, kStepKernelBlock, 0, st, p);
        else
            launch_plain(k_step<MODE, SM, 8, false>, nb, kStepKernelBlock, 0, st, p);
        break;
    case 16:
        if (lean)
            launch_plain(k_step<MODE, SM, 16, true>, nb, kStepKernelBlock, 0, st, p);
        else
            launch_plain(k_step<MODE, SM, 16, false>, nb, kStepKernelBlock, 0, st, p);
        break;
    default:
        // without the energy sums a smaller block costs nothing and ends its wave earlier (256 -> 128 threads:
        // calls of 20 steps at 100,000 particles 1,564 -> 1,557 us, of 10 at 300,007 2,390 -> 2,356 us; 64
        // threads 1,601 and 2,353)
        if (MODE == MODE_STEP && part && lean)
            launch_plain(k_step<MODE_STEP_PART, SM, 4, true>, np, kStepPartBlock, 0, st, p);
        else if (MODE == MODE_STEP && part)
            launch_plain(k_step<MODE_STEP_PART, SM, 4, false>, np, kStepPartBlock, 0, st, p);
        else if (lean)
            launch_plain(k_step<MODE, SM, 4, true>, nb, kStepKernelBlock, 0, st, p);
        else
            launch_plain(k_step<MODE, SM, 4, false>, nb, kStepKernelBlock, 0, st, p);
        break;
    }
}

// Burying of every particle into the current layout (bs_set_burying), from caller order.
__global__ void k_set_burying(Params p, const float *b)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id < p.n)
        p.bur[p.ctl->lbuf][p.inv[id]] = b[id];
}

int launch_set_burying(const Params &p, const float *b, cudaStream_t st)
{
    k_set_burying<<<(p.n + 255) / 256, 256, 0, st>>>(p, b);
    return 1;
}

// New charges into the current layout (bs_set_charges): the value and the charged flag that
// decides Coulomb list membership (the caller forces a list rebuild before the next step).
__global__ void k_set_charges(Params p, const float *q)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id < p.n)
    {
        const int lb = p.ctl->lbuf, slot = p.inv[id];
        p.chg[lb][slot] = q[id];
        const unsigned int f = p.flags[lb][slot] & ~static_cast<unsigned int>(PF_CHARGED);
        p.flags[lb][slot] = q[id] != 0.0f ? (f | PF_CHARGED) : f;
    }
}

int launch_set_charges(const Params &p, const float *q, cudaStream_t st)
{
    k_set_charges<<<(p.n + 255) / 256, 256, 0, st>>>(p, q);
    return 1;
}

__global__ void k_set_springs(Params p, int nnz, const unsigned int *sid, const float *k, const float *r0)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz)
        return;
    const unsigned int t = sid[e] >> 1; // 2 * spring + end
    if (k)
        const_cast<float *>(p.sp_k)[e] = k[t];
    if (r0)
        const_cast<float *>(p.sp_r0)[e] = r0[t];
}

int launch_set_springs(const Params &p, int nnz, const unsigned int *sid, const float *k, const float *r0, cudaStream_t st)
{
    k_set_springs<<<(nnz + 255) / 256, 256, 0, st>>>(p, nnz, sid, k, r0);
    return 1;
}

// Adds one particle's external force for the next step and marks it pending (bs_set_force).
__global__ void k_ext_add(Params p, long long i, float fx, float fy, float fz)
{
    p.ext[3 * i] += fx;
    p.ext[3 * i + 1] += fy;
    p.ext[3 * i + 2] += fz;
    p.ctl->ext_pending = 1;
}

int launch_ext_add(const Params &p, long long i, float fx, float fy, float fz, cudaStream_t st)
{
    k_ext_add<<<1, 1, 0, st>>>(p, i, fx, fy, fz);
    return 1;
}

// Frame recorder, after a step (and the bodies and the probe): a frame is due when the step
// count is a multiple of frame_every and its ring slot does not already hold it (a step that did
// not run leaves the count, so the frame is not written twice). k_frame_open marks the slot as
// being written; k_frame writes the positions in caller order straight into the mapped host ring
// (one thread per particle, coalesced), and its last block writes the header after a system-wide
// fence, so a reader that sees the header's sequence number sees the whole frame.
__device__ __forceinline__ bool frame_due(const Params &p, long long &seq, int &slot)
{
    const long long st = *(volatile const long long *)&p.ctl->steps;
    if (st <= 0 || st % p.frame_every != 0)
        return false;
    seq = st / p.frame_every;
    slot = static_cast<int>(seq % p.frame_cap);
    return *(volatile const long long *)&p.frame_hdr[slot].seq != seq;
}

__global__ void k_frame_open(Params p)
{
    pdl_enter();
    long long seq;
    int slot;
    if (!frame_due(p, seq, slot))
        return;
    *(volatile long long *)&p.frame_hdr[slot].seq = -1;
    __threadfence_system();
}

__global__ void __launch_bounds__(256) k_frame(Params p)
{
    pdl_enter();
    long long seq;
    int slot;
    // the header of this slot is -1 while the frame is written: the decision is the same in every
    // block, because only the last block of this launch changes it
    const long long st = *(volatile const long long *)&p.ctl->steps;
    if (st <= 0 || st % p.frame_every != 0)
        return;
    seq = st / p.frame_every;
    slot = static_cast<int>(seq % p.frame_cap);
    if (*(volatile const long long *)&p.frame_hdr[slot].seq != -1)
        return;
    Ctl *ctl = p.ctl;
    const float4 *pos = p.pos[ctl->sbuf];
    float *dst = p.frame_xyz + static_cast<size_t>(slot) * 3 * static_cast<size_t>(p.n);
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < p.n; id += gridDim.x * blockDim.x)
    {
        const float4 q = pos[p.inv[id]];
        dst[3 * static_cast<size_t>(id)] = q.x;
        dst[3 * static_cast<size_t>(id) + 1] = q.y;
        dst[3 * static_cast<size_t>(id) + 2] = q.z;
    }
    __threadfence_system();
    __syncthreads();
    __shared__ bool last;
    if (threadIdx.x == 0)
        last = atomicAdd(&ctl->done_frame, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x != 0)
        return;
    __threadfence_system();
    FrameHeader *h = p.frame_hdr + slot;
    h->step = st;
    for (int k = 0; k < 6; ++k)
        h->energies[k] = ctl->energies[k];
    __threadfence_system();
    *(volatile long long *)&h->seq = seq;
    ctl->done_frame = 0u;
}

int launch_step(const Params &p, int mode, cudaStream_t st)
{
    int launched = launch_step_only(p, mode, st);
    if (mode != MODE_FORCES && p.nbody > 0)
        launched += launch_rigid(p, st); // after the step kernel, on the same stream
    if (mode != MODE_FORCES && p.probe_on)
    {
        launch_plain(k_probe, 1, 1024, 0, st, p);
        launched += 1;
    }
    if (mode != MODE_FORCES && p.frame_every > 0)
    {
        launch_plain(k_frame_open, 1, 1, 0, st, p);
        launch_plain(k_frame, std::min((p.n + 255) / 256, 608), 256, 0, st, p);
        launched += 2;
    }
    return launched;
}

int launch_steps(const Params &p, int count, cudaStream_t st)
{
    int launched = 0;
    // Frames are recorded between two steps. A single step gains nothing from k_run, whose launch is the dearer one (us a
    // step and its energies, k_run and k_step: networks of 300 and 5,000 38.6 and 37.0, 39.1 and 37.2, Lennard-Jones
    // 5,000 43.0 and 40.3), unless a body's or the probe's part would be a kernel of its own (two bodies: 43.9 and 51.1).
    if (p.run_on && p.frame_every == 0 && (count > 1 || p.nbody > 0 || p.probe_on))
        for (int k = 0; k < count; k += kRunMaxSteps, ++launched)
            launch_run(p, std::min(kRunMaxSteps, count - k), st);
    else
        for (int k = 0; k < count; ++k)
            launched += launch_step(p, p.frame_every == 0 && k + 1 < count ? MODE_STEP_PART : MODE_STEP, st);
    return launched;
}

int launch_step_only(const Params &p, int mode, cudaStream_t st)
{
#define BS_STEP_CASE(SMV)                                                                                              \
    case SMV:                                                                                                          \
        if (mode != MODE_FORCES)                                                                                       \
            launch_step_lanes<MODE_STEP, SMV>(p, st, mode == MODE_STEP_PART);                                          \
        else                                                                                                           \
            launch_step_lanes<MODE_FORCES, SMV>(p, st, false);                                                                \
        break;
    switch (p.steric_mode)
    {
        BS_STEP_CASE(BS_STERIC_LINEAR)
        BS_STEP_CASE(BS_STERIC_LJ_12_6_AMBER)
        BS_STEP_CASE(BS_STERIC_LJ_8_6_LEWITT)
        BS_STEP_CASE(BS_STERIC_LJ_8_6_ZACHARIAS)
    default:
        break;
    }
#undef BS_STEP_CASE
    return 1;
}

cudaError_t load_step_kernels()
{
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, k_unsort);
}

int launch_unsort(const Params &p, int what, float *out3, cudaStream_t st)
{
    k_unsort<<<(p.n + 255) / 256, 256, 0, st>>>(p, what, out3);
    return 1;
}

int launch_set_positions(const Params &p, const float *xyz, const float *vel, cudaStream_t st, const float *lo)
{
    k_set_state<<<(p.n + 255) / 256, 256, 0, st>>>(p, xyz, vel, lo);
    return 1;
}

int launch_diag_cells(const Params &p, float cutoff, float skin, uint32_t need_flag, long long *out, cudaStream_t st)
{
    k_diag_cells<<<1, 1024, 0, st>>>(p, cutoff, skin, need_flag, out);
    return 1;
}

int launch_diag_pairs(const Params &p, int term, long long *out, unsigned long long *count, unsigned long long cap,
                      cudaStream_t st)
{
    k_diag_pairs<<<(p.n + kStepBlock - 1) / kStepBlock, kStepBlock, 0, st>>>(p, term, out, count, cap);
    return 1;
}

} // namespace bsg
