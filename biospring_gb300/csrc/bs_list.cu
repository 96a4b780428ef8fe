// bs_list.cu -- typed pair lists of a dense system from the cell grid.
//
// Lists: steric (every pair within its cutoff + skin, dynamic and static partners apart), Coulomb (both
// charged) and hydrophobic (both hydrophobic), minus the slot itself and, when springs are enabled, its
// spring partners (Particle.cpp:213-218).
//
// The grid edge is (cutoff + skin) / kGridDiv, so a particle's neighbours lie within kGridDiv cells in
// each direction. A block owns a group of kGridDiv^3 cells (grid-stride over the groups), its homes, and
// stages in shared memory the (3 kGridDiv)^2 x-runs of 3 kGridDiv cells that hold every neighbour of
// the group; each run is a contiguous range of slots. Staged candidates are cut into chunks of 32, and a
// bit matrix (home, chunk) says who is a neighbour of whom:
//   a. distances: one home a lane, the chunk's candidates broadcast from shared memory, two at a time in
//      packed FP32; a word collects the signs of r^2 - R^2 by a funnel shift each. Five instructions a
//      candidate for 32 homes;
//   b. the bits of a home itself and of its spring partners are cleared;
//   c. rows: a list's words are the matrix words and the chunk's mask of static, charged or hydrophobic
//      candidates; 4 to 16 threads a home walk them bit by bit.
// This is done once for every distinct list radius (once when the cutoffs are equal). A neighbourhood
// larger than the stage is walked in tiles of it, a group of more than kListHomes homes in batches.
// Rows come out in ascending slot order (runs ascend in z, then y; slots ascend within a run).
//
// Bound: instruction issue (69% of the slots at 100,000 particles): of the 145 us there some 65 us are
// distances, staging and clearing, the rest the walk of the bits. Measured (ncu, us a build; before: one
// home a warp, one candidate a lane in windows of the x-bounded runs, 200 M warp instructions, now 117 M):
// 100,000 particles 234 -> 145, 12,000 71 -> 44, 6,007 with three radii 50 -> 36. The rows by one warp a home,
// a word or an output window at a time, took 159; one or two threads a home 171 and 157.

#include <algorithm>

#include "bs_device.cuh"

namespace bsg
{
namespace
{

constexpr int kListWarps = 8;
constexpr int kListThreads = 32 * kListWarps;
constexpr int kListBlocks = 5;                  // resident blocks per SM
constexpr int kListResident = 152 * kListBlocks;
constexpr int kListFull = 152 * 4;              // blocks that fill the chip
constexpr int kListTile = 1536;                 // candidates staged at once
constexpr int kListChunks = kListTile / 32;
constexpr int kListHomes = 64;                  // homes of a batch
constexpr int kChunkPitch = 36;                 // floats: chunks read at once by half warps hit other banks
constexpr int kHeld = 2;                        // spring partners a thread holds
constexpr int kMatPitch = kListHomes + 1;

constexpr int kD = kGridDiv;        // neighbours lie within kD cells
constexpr int kG = kGridDiv;        // a block's group is kG^3 cells
constexpr int kRowsD = kG + 2 * kD; // staged runs per dimension (y, z)
constexpr int kRows = kRowsD * kRowsD;
static_assert(kRows > 32 && kRows <= 64 && kG * kG <= 32, "two runs a lane");

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}

// Bits of the chunk's candidates closer to the home (nx, ny, nz: its coordinates negated, twice) than
// the radius (mr2: -R^2, twice), candidate c in bit c. The same float operations as a scalar
// fma(dz, dz, fma(dy, dy, dx dx)) < R^2.
__device__ __forceinline__ unsigned int near_bits(const float *x, const float *y, const float *z, f32x2 nx, f32x2 ny,
                                                  f32x2 nz, f32x2 mr2)
{
    unsigned int bits = 0u;
#pragma unroll
    for (int c = 0; c < 32; c += 4)
    {
        const ulonglong2 vx = *reinterpret_cast<const ulonglong2 *>(x + c);
        const ulonglong2 vy = *reinterpret_cast<const ulonglong2 *>(y + c);
        const ulonglong2 vz = *reinterpret_cast<const ulonglong2 *>(z + c);
        const f32x2 ax[2] = {vx.x, vx.y}, ay[2] = {vy.x, vy.y}, az[2] = {vz.x, vz.y};
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            const f32x2 dx = add2(ax[h], nx), dy = add2(ay[h], ny), dz = add2(az[h], nz);
            const f32x2 d = add2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), mr2);
            bits = __funnelshift_l(static_cast<unsigned int>(d), bits, 1);
            bits = __funnelshift_l(static_cast<unsigned int>(d >> 32), bits, 1);
        }
    }
    return __brev(bits);
}

// Appends to the home's row of list L the candidates of chunks [c0, c1) whose matrix bit is set and whose
// mask bit is set (or, inverted, clear). E adjacent threads share a home and take their part of the
// chunks each: they count theirs, learn where they start, and write them; 16-bit offsets go out four at a
// time where the row's 8-byte words are wholly theirs (the last word of a row is padded, rows are a
// multiple of 8 entries long). All threads of the warp call it; cnt (shared) is the row's length before and
// after.
template <bool P16, int E>
__device__ __forceinline__ void emit(const PairList &L, bool on, int home, int c0, int c1,
                                     const unsigned int *mask, unsigned int flip, const unsigned int *mat, const int *slot,
                                     int &cnt)
{
    const int q = threadIdx.x % E;
    int own = 0;
    const unsigned int *m = mat + c0 * kMatPitch, *k = mask + c0;
    if (on)
        for (int c = c0; c < c1; ++c, m += kMatPitch, ++k)
            own += __popc(*m & (*k ^ flip));
    int inc = own;
#pragma unroll
    for (int o = 1; o < E; o <<= 1)
    {
        const int v = __shfl_up_sync(0xffffffffu, inc, o, E);
        if (q >= o)
            inc += v;
    }
    const int start = cnt; // every thread of the home has read it before the last of them writes it
    __syncwarp();
    if (on && q == E - 1)
        cnt = start + inc;
    int at = start + inc - own;
    const int end = min(at + own, L.cap);
    if (!on || at >= end)
        return;
    const size_t row = static_cast<size_t>(home) * L.cap;
    m = mat + c0 * kMatPitch;
    k = mask + c0;
    const int *sl = slot + 32 * c0 + 31;
    unsigned int w = *m & (*k ^ flip);
    if (P16)
    {
        short *out = reinterpret_cast<short *>(L.idx) + row;
        const int whole = (at + 3) & ~3;                       // the first word that is wholly this thread's
        const int tail = q == E - 1 ? INT_MAX : end & ~3;  // entries from here on go out one by one
        unsigned int lo = 0u, hi = 0u;                         // the last four entries
        while (at < end)
        {
            if (w == 0u)
            {
                m += kMatPitch;
                sl += 32;
                w = *m & (*++k ^ flip);
                continue;
            }
            const unsigned int low = w & (0u - w);
            const unsigned int off = static_cast<unsigned int>(sl[-__clz(low)] - home);
            w ^= low;
            lo = __funnelshift_r(lo, hi, 16);
            hi = __byte_perm(hi, off, 0x5432);
            ++at;
            if (at <= whole || at > tail)
                out[at - 1] = static_cast<short>(off);
            else if ((at & 3) == 0)
                *reinterpret_cast<uint2 *>(out + at - 4) = make_uint2(lo, hi);
        }
        if (q == E - 1 && (at & 3) && at > whole)
        {
            const int gap = 4 - (at & 3); // 1 to 3 entries of padding
            const unsigned long long v = ((static_cast<unsigned long long>(hi) << 32) | lo) >> (16 * gap);
            *reinterpret_cast<uint2 *>(out + (at & ~3)) =
                make_uint2(static_cast<unsigned int>(v), static_cast<unsigned int>(v >> 32));
        }
    }
    else
    {
        unsigned int *out = L.idx + row;
        while (at < end)
        {
            if (w == 0u)
            {
                m += kMatPitch;
                sl += 32;
                w = *m & (*++k ^ flip);
                continue;
            }
            const unsigned int low = w & (0u - w);
            out[at++] = static_cast<unsigned int>(sl[-__clz(low)]);
            w ^= low;
        }
    }
}

template <bool PL16, int SPLIT> __global__ void __launch_bounds__(kListThreads, kListBlocks) k_pairlist(Params p)
{
    pdl_enter();
    __shared__ int sh_first[kRows], sh_end[kRows], sh_off[kRows + 1]; // runs: slots, offset in the candidates
    __shared__ int sh_home[kG * kG][2];                               // the group's home x-runs: first slot, first home
    __shared__ __align__(16) float sh_x[kListChunks * kChunkPitch], sh_y[kListChunks * kChunkPitch],
        sh_z[kListChunks * kChunkPitch];
    __shared__ int sh_slot[kListTile];
    __shared__ unsigned int sh_static[kListChunks], sh_charged[kListChunks], sh_hydro[kListChunks];
    __shared__ unsigned int sh_mat[kListChunks * kMatPitch]; // [chunk][home]
    __shared__ float4 sh_hpos[kListHomes];
    __shared__ int sh_hslot[kListHomes];
    __shared__ unsigned int sh_hflag[kListHomes];
    __shared__ int sh_cnt[kListHomes][kLists];
    __shared__ int blocked, n_home;
    Ctl *ctl = p.ctl;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        blocked = (status_of(ctl) & kRebuildBlocking) != 0;
    __syncthreads();
    if (blocked)
        return;
    const int nx = ctl->gnx, ny = ctl->gny, nz = ctl->gnz;
    const int ngx = (nx + kG - 1) / kG, ngy = (ny + kG - 1) / kG, ngz = (nz + kG - 1) / kG;
    const int ngroups = ngx * ngy * ngz;
    const int sb = ctl->sbuf, lb = ctl->lbuf;
    const float4 *__restrict__ pos = p.pos[sb];
    const unsigned int *__restrict__ fl = p.flags[lb];
    const size_t stride = static_cast<size_t>(p.npad);
    int home = -1, deg = 0;
    unsigned int held[kHeld] = {};
    constexpr int E = 4 * SPLIT, kHomes = kListThreads / E;    // threads a home; homes of a batch
    const int hq = threadIdx.x / E, tq = threadIdx.x % E; // this thread's home of the batch, and which of its threads it is
    const bool whole = SPLIT == 1 || (ngroups >= kListFull && 24ll * ngroups > p.n);
    for (int item = blockIdx.x; item < (whole ? ngroups : ngroups * SPLIT); item += gridDim.x)
    {
        const int grp = whole ? item : item / SPLIT, part = item % SPLIT;
        const int gx0 = grp % ngx * kG, gy0 = grp / ngx % ngy * kG, gz0 = grp / (ngx * ngy) * kG;
        const int xa = max(gx0 - kD, 0), xb = min(gx0 + kG - 1 + kD, nx - 1), hxb = min(gx0 + kG - 1, nx - 1);
        __syncthreads(); // the previous group's tables are no longer read
        if (wid == 0)
        {
            // lane r: run r and run r + 32, and home run r
            int first[2] = {0, 0}, len[2] = {0, 0};
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int r = lane + 32 * h, y = gy0 - kD + r % kRowsD, z = gz0 - kD + r / kRowsD;
                if (r < kRows && y >= 0 && y < ny && z >= 0 && z < nz)
                {
                    const int base = (z * ny + y) * nx;
                    first[h] = p.cell_start[base + xa];
                    len[h] = p.cell_start[base + xb + 1] - first[h];
                }
            }
            int hfirst = 0, hlen = 0;
            if (lane < kG * kG)
            {
                const int y = gy0 + lane % kG, z = gz0 + lane / kG;
                if (y < ny && z < nz)
                {
                    const int base = (z * ny + y) * nx;
                    hfirst = p.cell_start[base + gx0];
                    hlen = p.cell_start[base + hxb + 1] - hfirst;
                }
            }
            // offsets of the runs, and for empty runs a first slot that keeps the slots ascending
            int base_off = 0, base_end = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                int inc = len[h], top = len[h] > 0 ? first[h] + len[h] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int a = __shfl_up_sync(0xffffffffu, inc, o), b = __shfl_up_sync(0xffffffffu, top, o);
                    if (lane >= o)
                    {
                        inc += a;
                        top = max(top, b);
                    }
                }
                top = max(top, base_end);
                const int r = lane + 32 * h;
                if (r < kRows)
                {
                    sh_first[r] = len[h] > 0 ? first[h] : top;
                    sh_end[r] = top;
                    sh_off[r] = base_off + inc - len[h];
                }
                base_off += __shfl_sync(0xffffffffu, inc, 31);
                base_end = __shfl_sync(0xffffffffu, top, 31);
            }
            int hinc = hlen;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int a = __shfl_up_sync(0xffffffffu, hinc, o);
                if (lane >= o)
                    hinc += a;
            }
            if (lane < kG * kG)
            {
                sh_home[lane][0] = hfirst;
                sh_home[lane][1] = hinc - hlen;
            }
            const int nh = __shfl_sync(0xffffffffu, hinc, 31);
            if (PL16 && nh > 0)
            {
                // every candidate offset of this group fits 16 bits, or the list goes 32-bit
                const int lo = __reduce_min_sync(0xffffffffu, min(len[0] > 0 ? first[0] : INT_MAX, len[1] > 0 ? first[1] : INT_MAX));
                const int hmin = __reduce_min_sync(0xffffffffu, hlen > 0 ? hfirst : INT_MAX);
                const int hmax = __reduce_max_sync(0xffffffffu, hlen > 0 ? hfirst + hlen : INT_MIN);
                if (lane == 0 && (base_end - 1 - hmin > 32767 || lo - (hmax - 1) < -32768))
                    atomicOr(&ctl->status, ST_WIDE);
            }
            if (lane == 0)
            {
                sh_off[kRows] = base_off;
                n_home = nh;
            }
        }
        __syncthreads();
        const int n_cand = sh_off[kRows];
        const int h0 = whole ? 0 : n_home * part / SPLIT, h1 = whole ? n_home : n_home * (part + 1) / SPLIT;
        for (int hb = h0; hb < h1; hb += kHomes)
        {
            const int nhb = min(kHomes, h1 - hb);
            for (int tile = 0; tile < n_cand; tile += kListTile)
            {
                const int nt = min(kListTile, n_cand - tile), chunks = (nt + 31) / 32;
                if (hb > h0 || tile > 0)
                    __syncthreads(); // the previous tile is no longer read
                // ---- the batch's homes, E threads each; their first spring partners are on the way while
                // the candidates are staged ----
                if (tile == 0)
                {
                    home = -1;
                    deg = 0;
                    if (hq < nhb)
                    {
                        int u = 0;
                        while (u + 1 < kG * kG && sh_home[u + 1][1] <= hb + hq)
                            ++u;
                        home = sh_home[u][0] + (hb + hq - sh_home[u][1]);
                        deg = p.spring_on ? p.se_deg[home] : 0;
                        if (tq == 0)
                        {
                            sh_hslot[hq] = home;
                            sh_hpos[hq] = pos[home];
                            sh_hflag[hq] = fl[home];
#pragma unroll
                            for (int q = 0; q < kLists; ++q)
                                sh_cnt[hq][q] = 0;
                        }
#pragma unroll
                        for (int u2 = 0; u2 < kHeld; ++u2)
                            if (tq + E * u2 < deg)
                                held[u2] = p.se_col[static_cast<size_t>(tq + E * u2) * stride + home] & kSlotMask;
                    }
                }
                // ---- candidates: a warp a chunk ----
                if (tile > 0 || hb == h0 || n_cand > kListTile)
                    for (int c = wid; c < chunks; c += kListWarps)
                    {
                        const int k = 32 * c + lane;
                        float4 q = make_float4(1.0e30f, 1.0e30f, 1.0e30f, 0.f); // past the end: far from every home
                        unsigned int f = 0u;
                        int slot = -1;
                        if (k < nt)
                        {
                            int a = 0, b = kRows - 1; // the last run whose offset is <= the candidate
                            while (a < b)
                            {
                                const int m = (a + b + 1) >> 1;
                                if (sh_off[m] <= tile + k)
                                    a = m;
                                else
                                    b = m - 1;
                            }
                            slot = sh_first[a] + (tile + k - sh_off[a]);
                            q = pos[slot];
                            f = fl[slot];
                        }
                        sh_x[c * kChunkPitch + lane] = q.x;
                        sh_y[c * kChunkPitch + lane] = q.y;
                        sh_z[c * kChunkPitch + lane] = q.z;
                        sh_slot[k] = slot | ((f & PF_STATIC) ? static_cast<int>(kEntryStatic) : 0);
                        const unsigned int ms = __ballot_sync(0xffffffffu, (f & PF_STATIC) != 0);
                        const unsigned int mc = __ballot_sync(0xffffffffu, (f & PF_CHARGED) != 0 || p.coul_all);
                        const unsigned int mh = __ballot_sync(0xffffffffu, (f & PF_HYDROPHOBIC) != 0);
                        if (lane == 0)
                        {
                            sh_static[c] = ms;
                            sh_charged[c] = mc;
                            sh_hydro[c] = mh;
                        }
                    }
                for (int cls = 0; cls < kTerms; ++cls)
                {
                    // the lists of one radius: those equal to list cls's, unless an earlier list has it too
                    if (!p.pl[cls].on)
                        continue;
                    const float r2 = p.pl[cls].r2;
                    bool seen = false;
                    for (int q = 0; q < cls; ++q)
                        seen = seen || (p.pl[q].on && p.pl[q].r2 == r2);
                    if (seen)
                        continue;
                    __syncthreads(); // the stage is complete, the previous radius's matrix no longer read
                    // ---- a. distances: sets of 32 homes, the last of 16 with two chunks at once if it fits ----
                    const f32x2 mr2 = pack2(-r2, -r2);
                    for (int set = 0; set < nhb; set += 32)
                    {
                        const bool half = nhb - set <= 16;
                        const int h = set + (half ? lane & 15 : lane);
                        const float4 q = h < nhb ? sh_hpos[h] : make_float4(-1.0e30f, -1.0e30f, -1.0e30f, 0.f);
                        const f32x2 hx = pack2(-q.x, -q.x), hy = pack2(-q.y, -q.y), hz = pack2(-q.z, -q.z);
                        const int per = half ? 2 : 1;
                        for (int c0 = wid * per; c0 < chunks; c0 += kListWarps * per)
                        {
                            const int c = min(half ? c0 + (lane >> 4) : c0, chunks - 1);
                            const unsigned int bits = near_bits(sh_x + c * kChunkPitch, sh_y + c * kChunkPitch,
                                                                sh_z + c * kChunkPitch, hx, hy, hz, mr2);
                            // (an odd last chunk is done by the lower half)
                            if (h < nhb && (!half || lane < 16 || c0 + 1 < chunks))
                                sh_mat[c * kMatPitch + h] = bits;
                        }
                    }
                    __syncthreads();
                    // ---- b. not a home's neighbours: itself and its spring partners ----
                    if (home >= 0)
                    {
                        auto clear = [&](const int j) {
                            int a = 0, b = kRows - 1; // the last run whose first slot is <= j
                            while (a < b)
                            {
                                const int m = (a + b + 1) >> 1;
                                if (sh_first[m] <= j)
                                    a = m;
                                else
                                    b = m - 1;
                            }
                            const int at = sh_off[a] + (j - sh_first[a]) - tile;
                            if (j >= sh_first[a] && j < sh_end[a] && at >= 0 && at < nt)
                                atomicAnd(&sh_mat[(at >> 5) * kMatPitch + hq], ~(1u << (at & 31)));
                        };
                        if (tq == 0)
                            clear(home);
#pragma unroll
                        for (int u = 0; u < kHeld; ++u)
                            if (tq + E * u < deg)
                                clear(static_cast<int>(held[u]));
                        for (int k = tq + E * kHeld; k < deg; k += E)
                            clear(static_cast<int>(p.se_col[static_cast<size_t>(k) * stride + home] & kSlotMask));
                    }
                    __syncthreads();
                    // ---- c. rows ----
                    {
                        const int h = hq, q = tq;
                        const int i = h < nhb ? sh_hslot[h] : 0;
                        const unsigned int fi = h < nhb ? sh_hflag[h] : PF_STATIC;
                        const bool dyn = !(fi & PF_STATIC);
                        const int c0 = chunks * q / E, c1 = chunks * (q + 1) / E; // this thread's chunks
                        const unsigned int *mat = sh_mat + h;
                        if (p.pl[0].on && p.pl[0].r2 == r2)
                        {
                            emit<PL16, E>(p.pl[0], dyn, i, c0, c1, sh_static, ~0u, mat, sh_slot, sh_cnt[h][0]);
                            if (p.pl[kListStericStatic].on)
                                emit<false, E>(p.pl[kListStericStatic], dyn, i, c0, c1, sh_static, 0u, mat, sh_slot,
                                            sh_cnt[h][kListStericStatic]);
                        }
                        if (p.pl[1].on && p.pl[1].r2 == r2)
                            emit<false, E>(p.pl[1], dyn && ((fi & PF_CHARGED) || p.coul_all), i, c0, c1, sh_charged, 0u, mat,
                                        sh_slot, sh_cnt[h][1]);
                        if (p.pl[2].on && p.pl[2].r2 == r2)
                            emit<false, E>(p.pl[2], dyn && (fi & PF_HYDROPHOBIC), i, c0, c1, sh_hydro, 0u, mat, sh_slot,
                                        sh_cnt[h][2]);
                    }
                }
            }
            __syncthreads(); // the counts of the batch are complete
            for (int k = threadIdx.x; k < nhb * kLists; k += kListThreads)
            {
                const int h = k / kLists, q = k % kLists, cap = p.pl[q].cap;
                int cnt = sh_cnt[h][q];
                if (cnt > cap)
                {
                    atomicOr(&ctl->status, ST_PAIR_CAPACITY);
                    atomicMax(&ctl->max_row[q], cnt);
                    cnt = cap;
                }
                p.pl[q].cnt[sh_hslot[h]] = cnt;
            }
        }
    }
}

} // namespace

template <int SPLIT> static void launch_split(const Params &p, cudaStream_t st)
{
    // The number of groups is only known on the device. A dense system (8 particles a group and more) has n / 8 at
    // most, or no more than the capacity: that many blocks, of which those past the last group return at once. One that
    // has spread out since has more, mostly empty ones: the blocks stride over them (12,000 particles eight times as far
    // apart, a block for each part of a group: 1,233 us a rebuild; so 246).
    cudaLaunchConfig_t cfg{};
    const int groups = std::min(p.cell_cap / (kGridDiv * kGridDiv * kGridDiv) + 1, std::max(p.n / 8, kListResident));
    cfg.gridDim = dim3(static_cast<unsigned>(SPLIT * groups));
    cfg.blockDim = dim3(kListThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (p.pl16)
        cudaLaunchKernelEx(&cfg, k_pairlist<true, SPLIT>, p);
    else
        cudaLaunchKernelEx(&cfg, k_pairlist<false, SPLIT>, p);
}

// A group's homes are split over 4 blocks up to 16,384 particles and over 2 up to 32,768: a block a
// group left half the SMs with one block or none at 6,000 particles. Measured (ncu, us a build, whole groups
// against split): 6,007 particles 57 -> 39, 12,000 46 -> 46 (2 parts 48). Where the particles have spread out, so that the
// groups alone fill the chip and hold fewer than 24 homes each, a block takes a whole group (us a rebuild, split against
// whole: 16,000 particles at 0.0244 per cubic A 1.4 times as far apart 86 -> 67, 1.7 times 98 -> 63; 24 homes are where the
// two meet: 1.2 times as far apart, 22 homes, 81 and 80).
int launch_pairlist(const Params &p, cudaStream_t st)
{
    if (p.n <= 16384)
        launch_split<4>(p, st);
    else if (p.n <= 32768)
        launch_split<2>(p, st);
    else
        launch_split<1>(p, st);
    return 1;
}

} // namespace bsg
