// bs_noalloc.cu -- nonbonded forces and energies of a small system by direct summation over all
// pairs, with every byte of scratch memory in one fixed-size array of this module, so that a call
// allocates nothing.
//
// Who needs it. A handle (bs_create/bs_setup) owns growable device buffers: pair lists, cell
// arrays, energy partials. Some callers cannot let a library allocate behind their back:
//   * a host application that manages all device memory through its own pool (a caching
//     allocator, a visualisation or steering front-end) and must keep its budget exact;
//   * an interactive loop that evaluates forces inside a fixed frame budget, where a device
//     allocation may synchronise the whole device and stall the frame;
//   * code that runs when the device is nearly full, where an allocation can fail at a point the
//     caller cannot recover from.
// Such callers pass device buffers they own; this entry point only reads and writes those and
// its own static scratch.
//
// The terms follow the reference force loop for one dynamic particle i
// (src/spn/SpringNetwork.cpp:93-198, src/spn/Particle.cpp:191-253, 269-330, 368-429):
// every other particle j within the term's cutoff acts on i; a dynamic partner's pair energy is
// shared half and half, a static partner's is counted in full at i; static particles get no
// force. Pair kernels: src/forcefield/energy/steric.hpp:27-156,
// electrostatic.hpp:16-49 (plus the eps = D r extension), hydrophobic.hpp:20-39.
// There is no spring topology here, so no pair is excluded: the result is the one a handle
// with spring.enable = 0 gives.

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "bs_common.cuh"

namespace bsg
{
namespace
{

constexpr int kNaMaxN = BS_NOALLOC_MAX_PARTICLES;
constexpr int kNaBlock = 256;                        // threads per block
constexpr int kNaHomes = 4;                          // home particles of a warp
constexpr int kNaMaxSplit = kNaBlock / 32;           // most warps that share a group of homes
constexpr int kNaMaxBlocks = 1280;                   // most blocks of a call (na_blocks)
constexpr int kNaTerms = 3;                          // steric, Coulomb, hydrophobic

// Scratch layout (byte offsets into na_scratch):
//   [kNaPosOff]  float4 [kNaMaxN]  x, y, z, steric factor P (the radius in linear mode)
//   [kNaPrmOff]  float4 [kNaMaxN]  steric factor F, charge, hydrophobicity, flag bits
//   [kNaBlkOff]  double [kNaMaxBlocks][kNaTerms]  per-block energy partials (overwritten)
//   [kNaDoneOff] unsigned int  blocks finished in the current call; must be 0 when a call
//                starts: set-up clears it, and the last block of every call puts it back to 0.
constexpr size_t kNaPosOff = 0;
constexpr size_t kNaPrmOff = kNaPosOff + sizeof(float4) * kNaMaxN;
constexpr size_t kNaBlkOff = kNaPrmOff + sizeof(float4) * kNaMaxN;
constexpr size_t kNaDoneOff = kNaBlkOff + sizeof(double) * kNaMaxBlocks * kNaTerms;
constexpr size_t kNaBytes = (kNaDoneOff + sizeof(unsigned int) + 255) / 256 * 256; // 555 KB

static __device__ __align__(256) unsigned char na_scratch[kNaBytes];

struct NaParams
{
    int n;
    int steric_on, coulomb_on, hydro_on;
    int steric_mode, dist_dielectric;
    float c_steric, c_coulomb, c_hydro;
    float lo2_s, hi2_s, lo2_c, hi2_c, lo2_h, hi2_h;
    float kf_steric, ke_steric;     // force and energy factors of each term
    float kf_elec, ke_elec;
    float kf_hydro, ke_hydro;
};

struct NaBuffers
{
    float4 *pos;
    float4 *prm;
    double *blk;
    unsigned int *done;
};

__host__ __device__ inline NaBuffers na_buffers(unsigned char *base)
{
    NaBuffers b;
    b.pos = reinterpret_cast<float4 *>(base + kNaPosOff);
    b.prm = reinterpret_cast<float4 *>(base + kNaPrmOff);
    b.blk = reinterpret_cast<double *>(base + kNaBlkOff);
    b.done = reinterpret_cast<unsigned int *>(base + kNaDoneOff);
    return b;
}

// The reference's pair test for one cutoff: FP64 distance of the float coordinates
// (nsearch.hpp:230), then the float-rounded FP64 norm of the float difference
// (Particle.cpp:222-224, measure.hpp:188-196). Called only inside a narrow band around the
// cutoff, where the FP32 squared distance cannot decide.
__device__ __noinline__ bool na_exact_in(float4 a, float4 b, float cutoff, bool nonzero)
{
    const double ax = __dsub_rn(static_cast<double>(a.x), static_cast<double>(b.x));
    const double ay = __dsub_rn(static_cast<double>(a.y), static_cast<double>(b.y));
    const double az = __dsub_rn(static_cast<double>(a.z), static_cast<double>(b.z));
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay)), __dmul_rn(az, az));
    if (!(__dsqrt_rn(s) < static_cast<double>(cutoff)))
        return false;
    const double fx = static_cast<double>(__fsub_rn(b.x, a.x));
    const double fy = static_cast<double>(__fsub_rn(b.y, a.y));
    const double fz = static_cast<double>(__fsub_rn(b.z, a.z));
    double nrm = 0.0;
    if (!(fabs(fx) < 1e-40 && fabs(fy) < 1e-40 && fabs(fz) < 1e-40))
        nrm = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(fx, fx), __dmul_rn(fy, fy)), __dmul_rn(fz, fz)));
    const float d = __double2float_rn(nrm);
    return d < cutoff && (!nonzero || d != 0.0f);
}

__device__ __forceinline__ bool na_in(float r2, float lo2, float hi2, float4 a, float4 b, float cutoff,
                                      bool nonzero)
{
    if (r2 >= hi2)
        return false;
    if (r2 < lo2 && r2 > 1e-20f)
        return true;
    return na_exact_in(a, b, cutoff, nonzero);
}

// Packs the caller's arrays into the scratch: per-particle steric factors of the combination
// rules (CombinationRules.hpp:18-31), so that a pair needs products only: Amber and Lewitt use
// sqrt(eps_i eps_j) (r_i r_j)^(k/2), P = sqrt(eps) r^3, F = sqrt(eps) r^6 (Amber) or r^4
// (Lewitt); Zacharias uses eps_i eps_j (r_i r_j)^k, P = eps r^6, F = eps r^8.
__global__ void __launch_bounds__(256) k_na_pack(NaParams p, const float *__restrict__ xyz,
                                                 const float *__restrict__ radius,
                                                 const float *__restrict__ epsilon,
                                                 const float *__restrict__ charge,
                                                 const float *__restrict__ hydro,
                                                 const uint8_t *__restrict__ is_static, NaBuffers b)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n)
        return;
    const double r = radius ? static_cast<double>(radius[i]) : 0.0;
    const double e = epsilon ? static_cast<double>(epsilon[i]) : 0.0;
    double P = r, F = 0.0;
    if (p.steric_mode == BS_STERIC_LJ_12_6_AMBER || p.steric_mode == BS_STERIC_LJ_8_6_LEWITT)
    {
        const double se = sqrt(e), r2 = r * r;
        P = se * r2 * r;
        F = p.steric_mode == BS_STERIC_LJ_12_6_AMBER ? se * (r2 * r2 * r2) : se * (r2 * r2);
    }
    else if (p.steric_mode == BS_STERIC_LJ_8_6_ZACHARIAS)
    {
        const double r2 = r * r, r6 = r2 * r2 * r2;
        P = e * r6;
        F = e * (r6 * r2);
    }
    const float q = charge ? charge[i] : 0.0f;
    const float h = hydro ? hydro[i] : 0.0f;
    unsigned int fl = 0u;
    if (is_static && is_static[i])
        fl |= PF_STATIC;
    if (q != 0.0f)
        fl |= PF_CHARGED;
    if (h != 0.0f)
        fl |= PF_HYDROPHOBIC;
    b.pos[i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], static_cast<float>(P));
    b.prm[i] = make_float4(static_cast<float>(F), q, h, __uint_as_float(fl));
}

// The pair terms of one home and one partner (steric.hpp, electrostatic.hpp, hydrophobic.hpp).
__device__ __forceinline__ void na_pair(const NaParams &p, float4 pi, float4 qi, float4 pj, float4 qj, float (&v)[6])
{
    float &fx = v[0], &fy = v[1], &fz = v[2], &es = v[3], &ec = v[4], &eh = v[5];
    const unsigned int fi = __float_as_uint(qi.w), fj = __float_as_uint(qj.w);
    const float w = (fj & PF_STATIC) ? 1.0f : 0.5f;
    const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    float f = 0.0f;
    if (p.steric_on && na_in(r2, p.lo2_s, p.hi2_s, pi, pj, p.c_steric, false))
    {
        float fod = 0.0f;
        if (p.steric_mode == BS_STERIC_LINEAR)
        {
            // E = (d - (ri + rj))^2 / 2 when overlapping, |F| = |d - (ri + rj)|
            const float d = sqrtf(r2);
            const float dv = d - (pi.w + pj.w);
            if (dv <= 0.0f)
            {
                fod = d > 0.0f ? dv / d : 0.0f;
                es = fmaf(w * 0.5f, dv * dv, es);
            }
        }
        else if (r2 >= 0.01f) // d < 0.1 A gives zero
        {
            const float inv2 = 1.0f / r2;
            const float i6 = inv2 * inv2 * inv2;
            const float t6 = pi.w * pj.w * i6;
            if (p.steric_mode == BS_STERIC_LJ_12_6_AMBER)
            {
                const float t12 = qi.x * qj.x * i6 * i6;
                es = fmaf(w, t12 - 2.0f * t6, es);
                fod = 12.0f * (t6 - t12) * inv2;
            }
            else if (p.steric_mode == BS_STERIC_LJ_8_6_LEWITT)
            {
                const float t8 = qi.x * qj.x * i6 * inv2;
                es = fmaf(w, 3.0f * t8 - 4.0f * t6, es);
                fod = 24.0f * (t6 - t8) * inv2;
            }
            else
            {
                const float t8 = qi.x * qj.x * i6 * inv2;
                es = fmaf(w, t8 - t6, es);
                fod = (6.0f * t6 - 8.0f * t8) * inv2;
            }
        }
        f = fod * p.kf_steric;
    }
    if (p.coulomb_on && (fi & fj & PF_CHARGED) && r2 >= 1e-6f &&
        na_in(r2, p.lo2_c, p.hi2_c, pi, pj, p.c_coulomb, true))
    {
        const float inv = 1.0f / sqrtf(r2);
        float tq = qi.y * qj.y * inv;
        float fod;
        if (p.dist_dielectric)
        {
            tq *= inv;
            fod = -2.0f * tq * inv * inv;
        }
        else
            fod = -tq * inv * inv;
        ec = fmaf(w, tq, ec);
        f = fmaf(fod, p.kf_elec, f);
    }
    if (p.hydro_on && (fi & fj & PF_HYDROPHOBIC) && na_in(r2, p.lo2_h, p.hi2_h, pi, pj, p.c_hydro, true))
    {
        const float d = sqrtf(r2);
        const float x = qi.z * qj.z * expf(-d);
        eh = fmaf(-w, x, eh);
        f = fmaf(x / d, p.kf_hydro, f);
    }
    fx = fmaf(dx, f, fx);
    fy = fmaf(dy, f, fy);
    fz = fmaf(dz, f, fz);
}

// All-pairs forces in two phases a warp. A warp owns kNaHomes home particles and runs through its
// share of the particles j, 32 at a time, one a lane: phase 1 tests each against every home with the
// FP32 squared distance alone and appends the accepted j to the home's queue (one ballot a home);
// phase 2 takes a home's next 32 queued partners, one a lane, and evaluates every term. Within the
// cutoffs of a dense system lie a few per cent of the particles, so evaluating in place would
// run the pair body for one or two lanes of the warp in most windows; through the queue it runs
// with all lanes busy, and the test, some 15 instructions for 32 pairs, is what bounds the kernel.
// `split` warps (1, 2, 4 or 8) share a group of homes, each taking every split-th window, so that
// small systems still fill the chip; the host picks it from n. The sums of the lanes and then
// of the split warps are added in a fixed order.
// Measured (pack and forces, us): one thread a particle in 64-thread blocks 139 / 798 / 2,285 at 500 /
// 4,001 / 16,384 particles (63 blocks of 2 warps on 152 SMs at 4,001), this form 17 / 44 / 260. The
// lanes' sums wait in shared memory: held in registers for four homes they took 118 of them, and
// 16 warps an SM left 56% of the issue slots without a ready warp.
__global__ void __launch_bounds__(kNaBlock, 3) k_na_forces(NaParams p, int split, float *__restrict__ forces,
                                                        double *__restrict__ energies, NaBuffers b)
{
    constexpr int R = kNaHomes, W = kNaBlock / 32;
    constexpr int NV = 6; // force x, y, z and three energies of a home
    __shared__ unsigned short sh_queue[W][R][64];
    __shared__ float4 sh_home[W][R];
    __shared__ float sh_acc[W][R][NV][32]; // each lane's sums, out of the registers of phase 1
    __shared__ float sh_sum[W][R][NV];
    __shared__ double sh_e[W][kNaTerms];
    __shared__ bool last;
    asm volatile("griddepcontrol.wait;" ::: "memory"); // the packed particles of k_na_pack
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = warp / split, part = warp % split; // home group in the block, share of its windows
    const int h0 = (blockIdx.x * (W / split) + group) * R;
    const unsigned int below = (1u << lane) - 1u;
    float hx[R], hy[R], hz[R];
    float r2max[R]; // 0: the home takes no pairs (static, past the end, or no term acts on it)
    bool any = false;
#pragma unroll
    for (int r = 0; r < R; ++r)
    {
        const int i = h0 + r;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        r2max[r] = 0.0f;
        if (i < p.n)
        {
            x = b.pos[i];
            const unsigned int fi = __float_as_uint(b.prm[i].w);
            if (!(fi & PF_STATIC))
            {
                float m = p.steric_on ? p.hi2_s : 0.0f;
                if (p.coulomb_on && (fi & PF_CHARGED))
                    m = fmaxf(m, p.hi2_c);
                if (p.hydro_on && (fi & PF_HYDROPHOBIC))
                    m = fmaxf(m, p.hi2_h);
                r2max[r] = m;
            }
        }
        hx[r] = x.x;
        hy[r] = x.y;
        hz[r] = x.z;
        if (lane == 0)
            sh_home[warp][r] = x;
#pragma unroll
        for (int q = 0; q < NV; ++q)
            sh_acc[warp][r][q][lane] = 0.0f;
        any = any || r2max[r] > 0.0f;
    }
    // queued partners of each home (low half) and the place of the first in its ring of 64 (high half)
    unsigned int fill[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
        fill[r] = 0u;
    // up to 32 queued partners of home r, one a lane; r is the same in every lane but no constant, so
    // that one copy of the pair body serves every home
    auto evaluate = [&](int r, int first, int m) {
        __syncwarp();
        const int i = h0 + r;
        const int j = lane < m ? sh_queue[warp][r][(first + lane) & 63] : i;
        if (j != i)
        {
            float v[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q)
                v[q] = sh_acc[warp][r][q][lane];
            na_pair(p, sh_home[warp][r], b.prm[i], b.pos[j], b.prm[j], v);
#pragma unroll
            for (int q = 0; q < NV; ++q)
                sh_acc[warp][r][q][lane] = v[q];
        }
        __syncwarp(); // the slots may be filled again
    };
    if (any)
    {
        const float nan = __int_as_float(0x7fffffff); // past the end: no distance compares
        const int step = 32 * split;
        int k = 32 * part + lane;
        float4 next = k < p.n ? b.pos[k] : make_float4(nan, nan, nan, 0.f);
        for (int k0 = 32 * part; k0 < p.n; k0 += step)
        {
            const float4 pj = next;
            const int j = k;
            k += step;
            next = k < p.n ? b.pos[k] : make_float4(nan, nan, nan, 0.f);
            unsigned int full = 0u;
#pragma unroll
            for (int r = 0; r < R; ++r)
            {
                const float dx = pj.x - hx[r], dy = pj.y - hy[r], dz = pj.z - hz[r];
                const float r2 = dx * dx + dy * dy + dz * dz;
                const bool in = r2 < r2max[r];
                const unsigned int m = __ballot_sync(0xffffffffu, in);
                if (in)
                    sh_queue[warp][r][((fill[r] >> 16) + fill[r] + __popc(m & below)) & 63] = static_cast<unsigned short>(j);
                fill[r] += __popc(m);
                full |= (fill[r] & 0x20u) << r; // 32 or more queued (at most 63)
            }
            if (full)
            {
#pragma unroll 1
                for (int r = 0; r < R; ++r)
                {
                    if (!((full >> r) & 0x20u))
                        continue;
                    unsigned int first = 0u;
#pragma unroll
                    for (int q = 0; q < R; ++q)
                        if (q == r)
                        {
                            first = fill[q] >> 16;
                            fill[q] += (32u << 16) - 32u;
                        }
                    evaluate(r, first, 32);
                }
            }
        }
#pragma unroll 1
        for (int r = 0; r < R; ++r)
        {
            unsigned int f = 0u;
#pragma unroll
            for (int q = 0; q < R; ++q)
                f = q == r ? fill[q] : f;
            if (f & 0xffffu)
                evaluate(r, f >> 16, f & 0xffffu);
        }
    }
    // The lanes' sums of every home and term: at each distance a lane passes on the half of its values that the
    // other keeps, so the values halve with the distance and lane 6 r + q ends with sum q of home r. The sums are those
    // of a shuffle tree a value, bit for bit, with 31 shuffles instead of 120
    // (us a call, before and now: 1 particle 12.4 and 10.4, 200 16.6 and 14.6, 4,001 49.8 and 43.8).
    {
        float v[32];
#pragma unroll
        for (int k = 0; k < 32; ++k)
            v[k] = k < R * NV ? sh_acc[warp][k / NV][k % NV][lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < o; ++k)
            {
                const float keep = (lane & o) ? v[k + o] : v[k], pass = (lane & o) ? v[k] : v[k + o];
                v[k] = keep + __shfl_xor_sync(0xffffffffu, pass, o);
            }
        if (lane < R * NV)
            sh_sum[warp][lane / NV][lane % NV] = v[0];
    }
    __syncthreads();
    // one thread a home adds the split warps' sums; energies go on in FP64, home by home
    if (part == 0 && lane < R)
    {
        float v[NV] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < split; ++s)
#pragma unroll
            for (int q = 0; q < NV; ++q)
                v[q] += sh_sum[warp + s][lane][q];
        const int i = h0 + lane;
        if (i < p.n)
        {
            forces[3 * i] = v[0];
            forces[3 * i + 1] = v[1];
            forces[3 * i + 2] = v[2];
        }
        double e[kNaTerms] = {static_cast<double>(v[3]) * p.ke_steric, static_cast<double>(v[4]) * p.ke_elec,
                              static_cast<double>(v[5]) * p.ke_hydro};
#pragma unroll
        for (int q = 0; q < kNaTerms; ++q)
        {
#pragma unroll
            for (int o = R / 2; o > 0; o >>= 1)
                e[q] += __shfl_down_sync((1u << R) - 1u, e[q], o, R);
            if (lane == 0)
                sh_e[group][q] = e[q];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
#pragma unroll
        for (int q = 0; q < kNaTerms; ++q)
        {
            double s = 0.0;
            for (int g = 0; g < W / split; ++g)
                s += sh_e[g][q];
            b.blk[blockIdx.x * kNaTerms + q] = s;
        }
        __threadfence();
        last = atomicAdd(b.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last)
        return;
    // the last block adds the blocks' energies: thread t takes blocks t, t + 256, ... in order, then
    // a fixed tree
    __threadfence();
    double tot[kNaTerms] = {0.0, 0.0, 0.0};
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += kNaBlock)
#pragma unroll
        for (int q = 0; q < kNaTerms; ++q)
            tot[q] += __ldcg(&b.blk[k * kNaTerms + q]);
#pragma unroll
    for (int q = 0; q < kNaTerms; ++q)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            tot[q] += __shfl_down_sync(0xffffffffu, tot[q], o);
        if (lane == 0)
            sh_e[warp][q] = tot[q];
    }
    __syncthreads();
    if (threadIdx.x < BS_NUM_ENERGIES)
    {
        const int q = threadIdx.x == BS_ENERGY_STERIC          ? 0
                      : threadIdx.x == BS_ENERGY_ELECTROSTATIC ? 1
                      : threadIdx.x == BS_ENERGY_HYDROPHOBIC   ? 2
                                                               : -1;
        double s = 0.0;
        if (q >= 0)
            for (int w = 0; w < W; ++w)
                s += sh_e[w][q];
        energies[threadIdx.x] = s;
    }
    if (threadIdx.x == 0)
        *b.done = 0u; // ready for the next call
}

// Warps that share a group of homes: 2 n warps up to 5,000 particles, n up to 10,000, n / 2 above, so 8,000 to 10,000
// at the upper ends (more than twice what the chip holds at once), so that the last blocks to finish are short; half as
// many homes a block cost more in part-filled queues than they gain. Measured (us a call, 2,500 / 5,000 / 10,000 /
// 16,384 particles): this rule 29 / 51 / 123 / 260, half the split 29 / 52 / 130 / 307.
constexpr int na_split(int n) { return n <= 5000 ? 8 : (n <= 10000 ? 4 : 2); }
constexpr int na_blocks(int n)
{
    const int homes = kNaHomes * (kNaMaxSplit / na_split(n));
    return (n + homes - 1) / homes;
}
static_assert(na_blocks(5000) <= kNaMaxBlocks && na_blocks(10000) <= kNaMaxBlocks && na_blocks(kNaMaxN) <= kNaMaxBlocks,
              "energy partials for every block");

float na_band_lo2(double c) { return static_cast<float>((c * (1.0 - 1.0 / 16384.0)) * (c * (1.0 - 1.0 / 16384.0))); }
float na_band_hi2(double c) { return static_cast<float>((c * (1.0 + 1.0 / 16384.0)) * (c * (1.0 + 1.0 / 16384.0))); }

void na_message(char *err, size_t len, const char *msg)
{
    if (err && len)
    {
        std::strncpy(err, msg, len - 1);
        err[len - 1] = '\0';
    }
}

// Scratch address per device, looked up once with that device current.
constexpr int kNaMaxDevices = 64;
std::mutex na_mutex;
unsigned char *na_ptr[kNaMaxDevices] = {};

} // namespace
} // namespace bsg

using namespace bsg;

extern "C" int bs_nonbonded_forces_noalloc(const bs_config *cfg, int64_t n, const float *d_xyz,
                                           const float *d_radius, const float *d_epsilon,
                                           const float *d_charge, const float *d_hydrophobicity,
                                           const uint8_t *d_is_static, float *d_forces, double *d_energies,
                                           void *stream, char *err, size_t err_len)
{
    char msg[192];
    if (!cfg || !d_xyz || !d_forces || !d_energies)
    {
        na_message(err, err_len, "null argument: cfg, xyz, forces and energies are required");
        return BS_E_ARG;
    }
    if (n < 1 || n > kNaMaxN)
    {
        std::snprintf(msg, sizeof msg, "particle count %lld outside [1, %d], the size of the static scratch",
                      static_cast<long long>(n), kNaMaxN);
        na_message(err, err_len, msg);
        return BS_E_ARG;
    }
    if (cfg->steric_enable)
    {
        if (!(cfg->steric_cutoff > 0.0))
        {
            na_message(err, err_len, "Steric cutoff must be > 0");
            return BS_E_ARG;
        }
        if (cfg->steric_mode < BS_STERIC_LINEAR || cfg->steric_mode > BS_STERIC_LJ_8_6_ZACHARIAS)
        {
            na_message(err, err_len, "unknown steric mode");
            return BS_E_ARG;
        }
        if (!d_radius || (cfg->steric_mode != BS_STERIC_LINEAR && !d_epsilon))
        {
            na_message(err, err_len, "steric term needs radius (and epsilon in the Lennard-Jones modes)");
            return BS_E_ARG;
        }
    }
    if (cfg->coulomb_enable && !(cfg->coulomb_cutoff > 0.0))
    {
        na_message(err, err_len, "Coulomb cutoff must be > 0");
        return BS_E_ARG;
    }
    if (cfg->coulomb_enable && !(cfg->coulomb_dielectric > 0.0))
    {
        na_message(err, err_len, "Coulomb dielectric must be > 0");
        return BS_E_ARG;
    }
    if (cfg->hydrophobicity_enable && !(cfg->hydrophobicity_cutoff > 0.0))
    {
        na_message(err, err_len, "Hydrophobicity cutoff must be > 0");
        return BS_E_ARG;
    }

    // Set-up, once per device: resolve the scratch address with that device current and clear
    // the block counter. The first call on a device does this (it loads this module onto the
    // device), so it should come before any stream capture.
    int dev = 0;
    cudaError_t rc = cudaGetDevice(&dev);
    if (rc != cudaSuccess || dev < 0 || dev >= kNaMaxDevices)
    {
        std::snprintf(msg, sizeof msg, "no usable current device (%s)", cudaGetErrorString(rc));
        na_message(err, err_len, msg);
        return BS_E_CUDA;
    }
    unsigned char *base = nullptr;
    {
        std::lock_guard<std::mutex> lock(na_mutex);
        if (!na_ptr[dev])
        {
            void *ptr = nullptr;
            rc = cudaGetSymbolAddress(&ptr, na_scratch);
            if (rc != cudaSuccess)
            {
                std::snprintf(msg, sizeof msg, "cudaGetSymbolAddress of the scratch failed: %s",
                              cudaGetErrorString(rc));
                na_message(err, err_len, msg);
                return BS_E_CUDA;
            }
            rc = cudaMemset(static_cast<unsigned char *>(ptr) + kNaDoneOff, 0, sizeof(unsigned int));
            if (rc == cudaSuccess)
                rc = cudaDeviceSynchronize();
            if (rc != cudaSuccess)
            {
                std::snprintf(msg, sizeof msg, "clearing the scratch counter failed: %s", cudaGetErrorString(rc));
                na_message(err, err_len, msg);
                return BS_E_CUDA;
            }
            na_ptr[dev] = static_cast<unsigned char *>(ptr);
        }
        base = na_ptr[dev];
    }

    NaParams p{};
    p.n = static_cast<int>(n);
    p.steric_on = cfg->steric_enable != 0;
    p.coulomb_on = cfg->coulomb_enable != 0 && d_charge != nullptr;
    p.hydro_on = cfg->hydrophobicity_enable != 0 && d_hydrophobicity != nullptr;
    p.steric_mode = cfg->steric_mode;
    p.dist_dielectric = cfg->dielectric_mode == BS_DIELECTRIC_DISTANCE;
    p.c_steric = static_cast<float>(cfg->steric_cutoff);
    p.c_coulomb = static_cast<float>(cfg->coulomb_cutoff);
    p.c_hydro = static_cast<float>(cfg->hydrophobicity_cutoff);
    p.lo2_s = na_band_lo2(p.c_steric);
    p.hi2_s = na_band_hi2(p.c_steric);
    p.lo2_c = na_band_lo2(p.c_coulomb);
    p.hi2_c = na_band_hi2(p.c_coulomb);
    p.lo2_h = na_band_lo2(p.c_hydro);
    p.hi2_h = na_band_hi2(p.c_hydro);
    const float kspring = static_cast<float>(kSpringForceConvert);
    p.kf_steric = kspring * static_cast<float>(cfg->steric_gridscale);
    p.ke_steric = static_cast<float>(cfg->steric_gridscale);
    const double D = cfg->coulomb_dielectric > 0.0 ? cfg->coulomb_dielectric : 1.0;
    p.kf_elec = static_cast<float>(kElecForceConvert / (4.0 * kPi) * cfg->coulomb_scale / D);
    p.ke_elec = static_cast<float>(kCoulombEnergyPerA * cfg->coulomb_scale / D);
    p.kf_hydro = kspring * static_cast<float>(cfg->hydrophobicity_scale);
    p.ke_hydro = static_cast<float>(kAvogadro * 1.0E-3) * static_cast<float>(cfg->hydrophobicity_scale);

    const NaBuffers b = na_buffers(base);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_na_pack<<<(p.n + 255) / 256, 256, 0, st>>>(p, d_xyz, d_radius, d_epsilon, d_charge, d_hydrophobicity,
                                                  d_is_static, b);
    // the force kernel starts launching while the packing runs and waits for it on the device
    const int split = na_split(p.n);
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(na_blocks(p.n));
    lc.blockDim = dim3(kNaBlock);
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    cudaLaunchKernelEx(&lc, k_na_forces, p, split, d_forces, d_energies, b);
    rc = cudaGetLastError();
    if (rc != cudaSuccess)
    {
        std::snprintf(msg, sizeof msg, "kernel launch failed: %s", cudaGetErrorString(rc));
        na_message(err, err_len, msg);
        return BS_E_CUDA;
    }
    return BS_OK;
}
