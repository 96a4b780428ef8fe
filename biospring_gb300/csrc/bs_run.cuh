// bs_run.cuh -- several steps of one system in one kernel (one translation unit per steric form: a process
// loads only the form it steps, and they compile side by side).
//
// A small system's step is latency, not work: a kernel a step pays the launch, the first reads of
// the control block and the parameters, and the energy reduction (two device-wide fences and
// counters in a row) for some 4 us of gathering. k_run is launched cooperatively, one thread group a
// particle as in k_step, and takes all steps up to the next list rebuild: between two steps stands one
// grid barrier (bodies take a second one), and the energies, which only the last step of a
// call can show, are reduced once, by that step's own partials. The particle's step is particle_step
// and the reduction reduce_energies, over the same blocks and in the same order as k_step's, so the
// results are the same bit for bit. The probe's reaction is summed block by block, and every block then
// computes the probe's step itself, so it costs no barrier of its own.
//
// Where registers allow, the lanes keep the first entries of their steric and spring rows from step to step:
// after a barrier, which empties the L1, each was a dependent read of its own. Calls with and without: Calpha
// network of 2,000 792 -> 706 us (2 blocks an SM; 729 with 3), training step of 10,000 4,507 -> 4,260 us (3
// blocks), Lennard-Jones 5,003 316 -> 304 us, 6,007 with the probe 510 -> 502 us.
//
// Bound: the chain of dependent loads of a step, then the barrier. Measured, a call of 50 to 100 steps
// with its rebuilds, a kernel a step against this one: Calpha network of 2,000 1,423 -> 905 us (100
// steps), Lennard-Jones beads 5,003 431 -> 339 us (20), receptor and ligand of 6,007 with the probe 677 ->
// 530 us (20), membrane of 20,000 with four bodies 1,460 -> 1,284 us (50).

#pragma once

#include <type_traits>

#include "bs_rigid.cuh"

namespace bsg
{
namespace
{

static_assert(kRigidBlock == kStepKernelBlock, "k_run's blocks serve the bodies");

// The probe's sum over this block's particles, (hi, lo) per axis, into the block's row of `part`.
__device__ __forceinline__ void probe_block_sum(const Params &p, const int first, const int count, float *part)
{
    // one warp an axis: 16 to 64 particles a block
    const int lane = threadIdx.x & 31, axis = threadIdx.x >> 5;
    __syncthreads();
    if (axis >= 3)
        return;
    float hi = 0.0f, lo = 0.0f;
    for (int s = first + lane; s < first + count; s += 32)
        ff_add(hi, lo, reinterpret_cast<const float *>(p.probe_f + s)[axis], 0.0f);
    warp_ff_sum(hi, lo);
    if (lane == 0)
    {
        part[2 * axis] = hi;
        part[2 * axis + 1] = lo;
    }
}

// The probe's own step from all blocks' sums (SpringNetwork.cpp:156-182), in every block alike, so
// that no second barrier has to publish it: position and velocity in `prb`, kinetic energy in `ke`.
__device__ __forceinline__ void probe_step(const Params &p, const float *part, float4 *prb, float *ke)
{
    __shared__ float sh_f[3];
    const int lane = threadIdx.x & 31, axis = threadIdx.x >> 5;
    if (axis < 3)
    {
        float hi = 0.0f, lo = 0.0f;
        for (unsigned int b = lane; b < gridDim.x; b += 32)
        {
            const float2 v = __ldcg(reinterpret_cast<const float2 *>(part + 8 * static_cast<size_t>(b) + 2 * axis));
            ff_add(hi, lo, v.x, v.y);
        }
        warp_ff_sum(hi, lo);
        if (lane == 0)
            sh_f[axis] = __fadd_rn(hi, lo);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        probe_advance(p, sh_f, prb[0], prb[1], *ke);
    __syncthreads();
}

// HOLD: the lanes keep the first entries of their rows in registers (RowHeld); 2 or 3 is also the blocks an SM
// that leave registers enough for it (128 or 80 a thread).
template <int SM, int T, bool LEAN, int HOLD>
__global__ void __launch_bounds__(kStepKernelBlock, HOLD ? HOLD : kStepMinBlocks) k_run(Params p, int count, float4 *save, float4 *save_lo)
{
    Ctl *ctl = p.ctl;
    if (status_of(ctl) != 0)
        return; // the same in every block: raised bits reach the status after the last barrier
    const int sb0 = ctl->sbuf, lb = ctl->lbuf;
    const bool ext = ctl->ext_pending != 0;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    constexpr int kPerBlock = kStepKernelBlock / T;
    __shared__ float4 prb[2]; // the probe's position and velocity
    __shared__ float probe_ke;
    const bool probe = !LEAN && p.probe_on;
    if (probe)
    {
        if (threadIdx.x == 0)
        {
            prb[0] = ctl->probe_pos;
            prb[1] = ctl->probe_vel;
        }
        __syncthreads();
    }
    using Held = std::conditional_t<HOLD != 0, RowHeld<T>, NoHeld>;
    const Held held = [&] {
        if constexpr (HOLD != 0)
            return RowHeld<T>(p, g / T, g % T, lb);
        else
            return NoHeld();
    }();
    float e[6];
    unsigned int gen = 0;
    int k = 0, go = 1;
    do
    {
#pragma unroll
        for (int q = 0; q < 6; ++q)
            e[q] = 0.0f;
        const int sb = sb0 ^ (k & 1);
        if (save && g % T == 0 && g / T < p.n)
        {
            const size_t at = static_cast<size_t>(k) * p.npad + g / T;
            save[at] = p.pos[sb][g / T];
            if (!LEAN && save_lo)
                save_lo[at] = p.pos_lo[sb][g / T];
        }
        int pend = particle_step<MODE_STEP, SM, T, true, LEAN, PosShared, Held>(p, g / T, g % T, p.n, sb, lb,
                                                                                 ext && k == 0, prb, e, held);
        float *part = p.run_probe + static_cast<size_t>(k & 1) * 8 * gridDim.x; // read until the next step's barrier
        if (probe)
        {
            const int first = blockIdx.x * kPerBlock;
            probe_block_sum(p, first, min(kPerBlock, p.n - first), part + 8 * static_cast<size_t>(blockIdx.x));
        }
        if (!LEAN && p.nbody > 0)
        {
            if (!grid_barrier(p, p.run_arrive, ++gen, 0)) // the bodies read every member's force
            {
                go = 0;
                break;
            }
            for (int b = blockIdx.x; b < p.nbody; b += gridDim.x)
            {
                pend |= rigid_body_step(p, b, sb);
                __syncthreads();
            }
        }
        if (pend)
            atomicOr(&ctl->status_pending, pend);
        ++k;
        if (k < count || probe)
        {
            go = grid_barrier(p, p.run_arrive, ++gen, pend);
            if (probe && go)
                probe_step(p, part, prb, &probe_ke);
        }
    } while (k < count && go == 1);
    if (go == 0)
    {
        if (threadIdx.x == 0)
            atomicOr(&ctl->status, ST_BARRIER);
        return;
    }
    if (!reduce_energies<6, kStepKernelBlock>(e, p.blk_energy, p.blk_cap, &ctl->done_step, ctl->energies))
        return;
    if (threadIdx.x == 0)
    {
        publish_energies(ctl);
        if (probe)
        {
            ctl->probe_pos = prb[0];
            ctl->probe_vel = prb[1];
            ctl->energies[BS_ENERGY_KINETIC] += static_cast<double>(probe_ke);
        }
        ctl->sbuf = sb0 ^ (k & 1);
        const long long steps = ctl->steps + k;
        ctl->steps = steps;
        ctl->rigid_steps = steps;
        ctl->probe_steps = steps;
        ctl->ext_pending = 0;
        *p.run_arrive = 0u; // every block has left its last barrier
        const int pend = atomicExch(&ctl->status_pending, 0);
        if (pend)
            atomicOr(&ctl->status, pend);
    }
}

template <int SM, int T, int HOLD> const void *run_lean(bool lean)
{
    return lean ? reinterpret_cast<const void *>(&k_run<SM, T, true, HOLD>)
                : reinterpret_cast<const void *>(&k_run<SM, T, false, HOLD>);
}

// The forms there are: with 16 lanes a particle the rows held at 2 or 3 blocks an SM, with 8 lanes at 3. With 4
// lanes the held entries are too small a part of the rows (a membrane of 20,000 got 2% slower).
template <int SM> const void *run_form(int lanes, bool lean, int hold)
{
    if (lanes == 16)
        return hold == 2 ? run_lean<SM, 16, 2>(lean) : (hold == 3 ? run_lean<SM, 16, 3>(lean) : run_lean<SM, 16, 0>(lean));
    if (lanes == 8)
        return hold == 2 ? nullptr : (hold == 3 ? run_lean<SM, 8, 3>(lean) : run_lean<SM, 8, 0>(lean));
    return lanes == 4 && hold == 0 ? run_lean<SM, 4, 0>(lean) : nullptr;
}

} // namespace
} // namespace bsg
