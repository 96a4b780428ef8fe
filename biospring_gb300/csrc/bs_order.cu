// bs_order.cu -- the first part of a list rebuild in one kernel: search grid, cell order of the
// particles, the state moved into it, the spring table of the new order. The pair lists follow
// (k_pairlist, k_batch_pairlist).
//
// k_order is launched cooperatively and strides over the particles, with a grid barrier between its
// phases:
//   1. bounding box (per system in an ensemble), the grid of the box
//   2. the cell of every particle and its place of arrival in the cell (one atomic)
//   3. exclusive scan of the cell counts: a share of the cells per block, totals first, then the starts
//   4. the order key (x coordinate, caller id) of every particle to its place in its cell
//   5. every particle counts the smaller keys of its cell, which gives its slot, and moves its state there:
//      reads in the old order, coalesced, scattered writes, no look-up of where a slot's particle was
//   6. the spring table, partners as slots
// With few cells (most systems of some thousand particles) phases 3 and 4 need no barrier: the key goes to a bin
// of its cell in phase 2, and every block scans all counts for itself (ncu: 2,000 particles 22.5 -> 18.4 us,
// 6,007 23.3 -> 18.9, 12,000 25.1 -> 21.1; with up to 12,288 cells scanned by every block 10,000 particles took
// 70 us instead of 27).
// The order within a cell is by x coordinate, ties by caller id: the layout is deterministic and every
// x-run of cells is one x-sorted sequence (the reference appends to a cell in index order,
// nsearch.hpp:376-389, an order no result here depends on).
//
// Bound: latency of the phases at small sizes (some loads and a barrier of about a microsecond each),
// scattered writes of the state and of the spring table at large ones. Measured (ncu, us, the chain of nine
// kernels this replaced against it): 2,000 particles 56 -> 23, 5,003 53 -> 24, 12,000 55 -> 25, 100,000 96 ->
// 44, ensemble of 64 systems with 228,000 particles 202 -> 90 (one warp a system had read its neighbours' cell
// counts one after the other, and one thread all systems').

#include <algorithm>

#include "bs_device.cuh"

namespace bsg
{
namespace
{

constexpr int kOrderBlock = 256;
constexpr int kOrderWarps = kOrderBlock / 32;
constexpr int kOrderScan = 4 * kOrderBlock; // cells of one pass of a block's share
// Single systems of few cells take a shorter way: keys go to a bin of their cell at once, and every block scans
// all counts for itself.
constexpr int kSmallCells = 4 * kOrderScan; // four a thread in four passes, starts as 16 bits in shared memory
constexpr int kSmallN = 65536;
constexpr int kBin = 64;           // keys of a cell's bin; a fuller cell sends the rebuild the long way
constexpr int kMaxSysCells = 1 << 26;       // a system spread wider than this falls back to one cell

// ref_cell_coord, from a float estimate unless that lies within its error of a whole number: the cell
// origin is a float, so x - origin and the product are within 3e-7 relative.
__device__ __forceinline__ int cell_coord(float x, double mn, float mnf, float inv, float radius, int ncell)
{
    const float t = (x - mnf) * inv;
    if (!(fabsf(t - rintf(t)) >= 1e-3f + 1e-6f * fabsf(t)))
        return ref_cell_coord(x, mn, radius, ncell);
    return t > 0.0f ? min(static_cast<int>(t), ncell - 1) : ref_cell_coord(x, mn, radius, ncell);
}

// A box as order-preserving codes: (min x, y, z) by atomicMin, (max x, y, z) by atomicMax.
__device__ __forceinline__ void box_merge(unsigned int *enc, const float (&v)[6])
{
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        atomicMin(&enc[k], f2ord(v[k]));
        atomicMax(&enc[3 + k], f2ord(-v[3 + k]));
    }
}

__device__ __forceinline__ void box_add(float (&v)[6], float4 q)
{
    v[0] = fminf(v[0], q.x);
    v[1] = fminf(v[1], q.y);
    v[2] = fminf(v[2], q.z);
    v[3] = fminf(v[3], -q.x);
    v[4] = fminf(v[4], -q.y);
    v[5] = fminf(v[5], -q.z);
}

__device__ __forceinline__ void box_warp_min(float (&v)[6])
{
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
}

// Exclusive prefix of v over the block's threads; the total in `total`.
__device__ __forceinline__ int block_scan(int v, int *sh, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o)
            inc += t;
    }
    __syncthreads();
    if (lane == 31)
        sh[warp] = inc;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kOrderWarps; ++w)
    {
        before += w < warp ? sh[w] : 0;
        total += sh[w];
    }
    return before + inc - v;
}

// Grid of system b of an ensemble from its box. A system spread too wide gets one cell: the neighbour
// walk then sees every particle, which gives the same pairs (every candidate is tested against the
// list radius).
__device__ __forceinline__ int system_grid(const Params &p, int b)
{
    unsigned int *enc = p.sys_box + 6 * static_cast<size_t>(b);
    const int n = p.sys_start[b + 1] - p.sys_start[b];
    float mn[3], mx[3];
    bool ok = n > 0;
    for (int k = 0; k < 3; ++k)
    {
        mn[k] = ord2f(__ldcg(enc + k));
        mx[k] = ord2f(__ldcg(enc + 3 + k));
        ok = ok && isfinite(mn[k]) && isfinite(mx[k]) && mn[k] <= mx[k];
        enc[k] = 0xffffffffu; // for the next rebuild
        enc[3 + k] = 0u;
    }
    SysGrid g;
    g.radius = p.list_radius / static_cast<float>(kSparseDiv);
    int nc[3] = {1, 1, 1};
    double gmin[3] = {0.0, 0.0, 0.0};
    double cells = !ok           ? 1.0
                   : p.lists_off ? free_grid_dims(mn, mx, g.radius, free_cells(n), gmin, nc)
                                 : grid_dims(mn, mx, g.radius, gmin, nc);
    if (!(cells <= static_cast<double>(kMaxSysCells)))
    {
        nc[0] = nc[1] = nc[2] = 1;
        cells = 1.0;
    }
    for (int k = 0; k < 3; ++k)
        g.gmin[k] = gmin[k];
    g.nx = nc[0];
    g.ny = nc[1];
    g.nz = nc[2];
    g.cells = static_cast<int>(cells);
    p.sys_grid[b] = g;
    p.stale_at[b] = LLONG_MAX; // a fresh list
    p.sys_status[b] &= ~ST_STALE;
    return g.cells;
}

template <bool BATCH>
__global__ void __launch_bounds__(kOrderBlock, 4) k_order(Params p)
{
    pdl_enter();
    Ctl *ctl = p.ctl;
    if (status_of(ctl) & kRebuildBlocking)
        return; // the same in every block: such a bit is raised after the first barrier, or by a later kernel
    __shared__ int sh[kOrderWarps];
    __shared__ float sh_box[kOrderWarps][6];
    __shared__ SysGrid sh_grid;
    __shared__ unsigned short sh_start[BATCH ? 1 : kSmallCells + 8];
    const int sb = ctl->sbuf, lb = ctl->lbuf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int me = blockIdx.x * kOrderBlock + threadIdx.x, threads = gridDim.x * kOrderBlock;
    const float4 *pos = p.pos[sb];
    unsigned int gen = 0;
    auto meet = [&]() {
        const bool ok = grid_barrier(p, p.order_sync, ++gen, 0) != 0;
        if (!ok && threadIdx.x == 0)
            atomicOr(&ctl->status, ST_BARRIER);
        return ok;
    };

    // ---- 1. boxes and grids ----
    {
        float v[6] = {FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX}; // min x,y,z and -max x,y,z
        if (BATCH)
        {
            // a warp takes a contiguous share, so its lanes are in one system nearly always
            const int warps = threads / 32, share = (p.n + 32 * warps - 1) / (32 * warps) * 32;
            const int i0 = (me / 32) * share, i1 = min(p.n, i0 + share);
            int cur = -1; // the system the box so far belongs to
            for (int i = i0 + lane; i < i0 + share; i += 32)
            {
                const int b = i < i1 ? p.sys_of[i] : -1;
                const int first = __shfl_sync(0xffffffffu, b, 0);
                const bool one = __all_sync(0xffffffffu, b == first || b < 0);
                if (first < 0)
                    break; // past the end: lane 0 holds the lowest index
                if (cur >= 0 && (first != cur || !one))
                {
                    box_warp_min(v);
                    if (lane == 0)
                        box_merge(p.sys_box + 6 * static_cast<size_t>(cur), v);
#pragma unroll
                    for (int k = 0; k < 6; ++k)
                        v[k] = FLT_MAX;
                    cur = -1;
                }
                if (b >= 0)
                    box_add(v, pos[i]);
                if (one)
                    cur = first;
                else
                {
                    if (b >= 0)
                        box_merge(p.sys_box + 6 * static_cast<size_t>(b), v);
#pragma unroll
                    for (int k = 0; k < 6; ++k)
                        v[k] = FLT_MAX;
                }
            }
            if (cur >= 0)
            {
                box_warp_min(v);
                if (lane == 0)
                    box_merge(p.sys_box + 6 * static_cast<size_t>(cur), v);
            }
        }
        else
        {
            for (int i = me; i < p.n; i += threads)
                box_add(v, pos[i]);
            box_warp_min(v);
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    sh_box[warp][k] = v[k];
            __syncthreads();
            if (threadIdx.x < 6)
            {
                float m = sh_box[0][threadIdx.x];
                for (int w = 1; w < kOrderWarps; ++w)
                    m = fminf(m, sh_box[w][threadIdx.x]);
                if (threadIdx.x < 3)
                    atomicMin(&ctl->bbox_enc[threadIdx.x], f2ord(m));
                else
                    atomicMax(&ctl->bbox_enc[threadIdx.x], f2ord(-m));
            }
        }
    }
    if (!meet())
        return;
    int nc; // cells, of all systems
    if (BATCH)
    {
        // block 0 makes the systems' grids and numbers their cells; a second barrier publishes them
        if (blockIdx.x == 0)
        {
            long long base = 0;
            for (int b0 = 0; b0 < p.nsys; b0 += kOrderBlock)
            {
                const int b = b0 + threadIdx.x;
                const int c = b < p.nsys ? system_grid(p, b) : 0;
                // at most 256 systems of 2^26 cells: the scan is in units that cannot overflow
                int total;
                const int lo = block_scan(c & 0xffff, sh, total);
                const long long lot = total;
                const long long at = base + lo + 65536ll * block_scan(c >> 16, sh, total);
                if (b < p.nsys)
                    p.sys_cells[b] = static_cast<int>(at < INT_MAX ? at : INT_MAX);
                base += lot + 65536ll * total;
            }
            if (threadIdx.x == 0)
            {
                const int total = static_cast<int>(base < INT_MAX ? base : INT_MAX);
                p.sys_cells[p.nsys] = total;
                ctl->gnx = min(total, p.cell_cap);
                ctl->gny = 1;
                ctl->gnz = 1;
                atomicAnd(&ctl->status, ~ST_STALE);
            }
        }
        if (!meet())
            return;
        nc = __ldcg(p.sys_cells + p.nsys);
    }
    else
    {
        // every block computes the grid; block 0 publishes it and resets the box after the next barrier
        if (threadIdx.x == 0)
        {
            float mn[3], mx[3];
            for (int k = 0; k < 3; ++k)
            {
                mn[k] = ord2f(__ldcg(&ctl->bbox_enc[k]));
                mx[k] = ord2f(__ldcg(&ctl->bbox_enc[3 + k]));
            }
            // the cell-block list build uses cells of a kGridDiv-th of the list radius, the
            // warp-per-particle build (sparse systems) cells of the list radius
            float edge = p.list_radius / static_cast<float>(p.pl_sparse ? kSparseDiv : kGridDiv);
            int dims[3];
            double gmin[3];
            double cells = p.lists_off ? free_grid_dims(mn, mx, edge, free_cells(p.n), gmin, dims)
                                       : grid_dims(mn, mx, edge, gmin, dims);
            if (!(mn[0] <= mx[0] && mn[1] <= mx[1] && mn[2] <= mx[2]))
            {
                // no particle has a coordinate: one cell for all, the step reports them
                dims[0] = dims[1] = dims[2] = 1;
                gmin[0] = gmin[1] = gmin[2] = 0.0;
                cells = 1.0;
            }
            for (int k = 0; k < 3; ++k)
                sh_grid.gmin[k] = gmin[k];
            sh_grid.radius = edge;
            sh_grid.nx = dims[0];
            sh_grid.ny = dims[1];
            sh_grid.nz = dims[2];
            sh_grid.cells = cells < 2.0e9 ? static_cast<int>(cells) : INT_MAX;
            if (blockIdx.x == 0)
            {
                for (int k = 0; k < 3; ++k)
                    ctl->gmin[k] = gmin[k];
                ctl->gradius = edge;
                ctl->gnx = dims[0];
                ctl->gny = dims[1];
                ctl->gnz = dims[2];
                if (status_of(ctl) & ST_STALE)
                    ctl->stale_events += 1;
                atomicAnd(&ctl->status, ~ST_STALE);
            }
        }
        __syncthreads();
        nc = sh_grid.cells;
    }
    const bool fits = nc <= p.cell_cap;
    if (!fits && blockIdx.x == 0 && threadIdx.x == 0)
    {
        ctl->ncells_needed = nc;
        atomicOr(&ctl->status, ST_CELL_CAPACITY);
    }
    if (!fits)
        nc = 0;

    auto order_key = [&](float x, int id) {
        return (static_cast<unsigned long long>(f2ord(x)) << 32) | static_cast<unsigned int>(id);
    };
    bool small = !BATCH && fits && nc <= kSmallCells && p.n < kSmallN;

    // ---- 2. cells and places of arrival ----
    if (fits)
        for (int i = me; i < p.n; i += threads)
        {
            const float4 q = pos[i];
            int base = 0;
            const SysGrid *g = &sh_grid;
            if (BATCH)
            {
                const int b = p.sys_of[i];
                base = p.sys_cells[b];
                g = p.sys_grid + b;
            }
            const float r = g->radius, inv = __frcp_rn(r);
            const int nx = g->nx, ny = g->ny;
            const double mx = g->gmin[0], my = g->gmin[1], mz = g->gmin[2];
            const int cx = cell_coord(q.x, mx, static_cast<float>(mx), inv, r, nx);
            const int cy = cell_coord(q.y, my, static_cast<float>(my), inv, r, ny);
            const int cz = cell_coord(q.z, mz, static_cast<float>(mz), inv, r, g->nz);
            const int c = base + cx + cy * nx + cz * nx * ny;
            const int at = atomicAdd(&p.cell_cnt[c], 1);
            p.cell_at[i] = make_int2(c, at);
            if (small && at < kBin)
                p.cell_bin[static_cast<size_t>(c) * kBin + at] = order_key(q.x, p.perm[lb][i]);
            else if (small)
                atomicOr(p.order_sync + 2, 1u);
        }
    if (!meet())
        return;
    if (!BATCH && blockIdx.x == 0 && threadIdx.x < 6)
        ctl->bbox_enc[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u; // every block has read the box
    small = small && __ldcg(p.order_sync + 2) == 0u;

    // A particle's slot, from the keys of its cell, and its state into it.
    auto move = [&](int i, int c, int s0, int len, const unsigned long long *keys) {
        const float4 q = pos[i], vel = p.vel[sb][i], prm = p.iprm[lb][i];
        const int id = p.perm[lb][i];
        const float fhi = p.fhi[lb][i], chg = p.chg[lb][i], hyd = p.hyd[lb][i];
        const unsigned int flags = p.flags[lb][i];
        const unsigned long long key = order_key(q.x, id);
        int s = s0;
#pragma unroll 4
        for (int f = 0; f < len; ++f)
            s += keys[f] < key;
        p.pos[sb ^ 1][s] = q;
        p.pos_build[s] = q;
        p.vel[sb ^ 1][s] = vel;
        if (p.pos_lo[0])
            p.pos_lo[sb ^ 1][s] = p.pos_lo[sb][i];
        p.fhi[lb ^ 1][s] = fhi;
        p.chg[lb ^ 1][s] = chg;
        p.hyd[lb ^ 1][s] = hyd;
        if (p.bur[0])
            p.bur[lb ^ 1][s] = p.bur[lb][i];
        p.flags[lb ^ 1][s] = flags;
        p.iprm[lb ^ 1][s] = prm;
        p.perm[lb ^ 1][s] = id;
        p.cell_of[s] = c;
        p.inv[id] = s;
    };
    if (small)
    {
        // ---- 3 to 5, few cells: every block scans the counts, and ranks from the bins ----
        int4 v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
        {
            // (counts past nc are zero; the array has room for a whole word at its end)
            const int c = t * kOrderScan + 4 * static_cast<int>(threadIdx.x);
            v[t] = c < nc ? __ldcg(reinterpret_cast<const int4 *>(p.cell_cnt + c)) : make_int4(0, 0, 0, 0);
        }
        int run = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t)
        {
            if (t * kOrderScan >= nc)
                break;
            const int c = t * kOrderScan + 4 * static_cast<int>(threadIdx.x);
            int total;
            const int at = run + block_scan(v[t].x + v[t].y + v[t].z + v[t].w, sh, total);
            run += total;
            sh_start[c] = static_cast<unsigned short>(at);
            sh_start[c + 1] = static_cast<unsigned short>(at + v[t].x);
            sh_start[c + 2] = static_cast<unsigned short>(at + v[t].x + v[t].y);
            sh_start[c + 3] = static_cast<unsigned short>(at + v[t].x + v[t].y + v[t].z);
        }
        __syncthreads();
        if (threadIdx.x == 0)
            sh_start[nc] = static_cast<unsigned short>(p.n);
        __syncthreads();
        for (int c = me; c <= nc; c += threads)
            p.cell_start[c] = sh_start[c];
        for (int i = me; i < p.n; i += threads)
        {
            const int c = p.cell_at[i].x, s0 = sh_start[c];
            move(i, c, s0, sh_start[c + 1] - s0, p.cell_bin + static_cast<size_t>(c) * kBin);
        }
        if (!meet())
            return;
        for (int c = me; c < nc; c += threads)
            p.cell_cnt[c] = 0; // for the next rebuild
    }
    else
    {

    // ---- 3. cell starts ----
    const int passes = (nc + kOrderScan * gridDim.x - 1) / (kOrderScan * static_cast<int>(gridDim.x));
    const int first = static_cast<int>(blockIdx.x) * passes * kOrderScan;
    if (fits)
    {
        int sum = 0;
        for (int c = first + threadIdx.x; c < min(nc, first + passes * kOrderScan); c += kOrderBlock)
            sum += __ldcg(p.cell_cnt + c);
        int total;
        block_scan(sum, sh, total);
        if (threadIdx.x == 0)
            p.tile_sum[blockIdx.x] = total;
    }
    if (!meet())
        return;
    if (fits)
    {
        int sum = 0, run;
        for (int b = threadIdx.x; b < static_cast<int>(blockIdx.x); b += kOrderBlock)
            sum += __ldcg(p.tile_sum + b);
        block_scan(sum, sh, run);
        for (int c0 = first; c0 < min(nc, first + passes * kOrderScan); c0 += kOrderScan)
        {
            const int c = c0 + 4 * static_cast<int>(threadIdx.x);
            int v[4], own = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                v[k] = c + k < nc ? __ldcg(p.cell_cnt + c + k) : 0;
                own += v[k];
            }
            int total, at = run + block_scan(own, sh, total);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (c + k < nc)
                {
                    p.cell_start[c + k] = at;
                    p.cell_cnt[c + k] = 0; // for the next rebuild
                    at += v[k];
                }
            run += total;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0)
            p.cell_start[nc] = p.n;
    }
    if (!meet())
        return;

    // ---- 4. keys, cell by cell ----
    if (fits)
        for (int i = me; i < p.n; i += threads)
        {
            const int2 at = p.cell_at[i];
            p.tmp_key[p.cell_start[at.x] + at.y] = order_key(pos[i].x, p.perm[lb][i]);
        }
    if (!meet())
        return;

    // ---- 5. slots; the state moves ----
    if (fits)
        for (int i = me; i < p.n; i += threads)
        {
            const int c = p.cell_at[i].x, s0 = p.cell_start[c];
            move(i, c, s0, p.cell_start[c + 1] - s0, p.tmp_key + s0);
        }
    if (!meet())
        return;
    }
    if (fits && blockIdx.x == 0 && threadIdx.x == 0)
    {
        ctl->sbuf = sb ^ 1;
        ctl->lbuf = lb ^ 1;
    }

    // ---- 6. springs, partners as slots (ELL, column-major): ell_lanes consecutive threads share a slot
    // and take every ell_lanes-th spring of its caller-order row; with one lane a slot the threads of a warp
    // store each column contiguously. U springs a pass, so that their look-ups overlap ----
    if (fits)
    {
        constexpr int U = 4;
        const int L = p.ell_lanes;
        const size_t stride = static_cast<size_t>(p.npad);
        const int *perm = p.perm[lb ^ 1];
        for (long long g = me; g < static_cast<long long>(p.npad) * L; g += threads)
        {
            const int s = static_cast<int>(g / L), t = static_cast<int>(g % L);
            if (s >= p.n)
            {
                if (t == 0)
                    p.se_deg[s] = 0;
                continue;
            }
            const int id = perm[s];
            const int r0 = p.sp_row[id], r1 = p.sp_row[id + 1];
            for (int e0 = r0 + t; e0 < r1; e0 += U * L)
            {
                unsigned int c[U], sid[U];
                float k[U], r[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    const int e = min(e0 + u * L, r1 - 1);
                    c[u] = __ldg(p.sp_col + e);
                    k[u] = __ldg(p.sp_k + e);
                    r[u] = __ldg(p.sp_r0 + e);
                    sid[u] = p.se_sid ? __ldg(p.sp_sid + e) : 0u;
                }
                unsigned int slot[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                    slot[u] = static_cast<unsigned int>(p.inv[c[u] & kSlotMask]);
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    const int e = e0 + u * L;
                    if (e >= r1)
                        break;
                    const size_t dst = static_cast<size_t>(e - r0) * stride + s;
                    p.se_col[dst] = slot[u] | (c[u] & ~kSlotMask);
                    p.se_k[dst] = k[u];
                    p.se_r0[dst] = r[u];
                    if (p.se_sid)
                        p.se_sid[dst] = sid[u];
                }
            }
            if (t == 0)
                p.se_deg[s] = r1 - r0;
        }
    }
    // the last block to finish: every block has left its last barrier
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(p.order_sync + 1, 1u) == gridDim.x - 1)
    {
        p.order_sync[0] = 0u;
        p.order_sync[1] = 0u;
        p.order_sync[2] = 0u;
    }
}

const void *order_fn(const Params &p)
{
    return p.nsys > 0 ? reinterpret_cast<const void *>(&k_order<true>) : reinterpret_cast<const void *>(&k_order<false>);
}

} // namespace

size_t order_bins(const Params &p)
{
    return p.n >= kSmallN ? 0 : static_cast<size_t>(std::min(p.cell_cap, kSmallCells)) * kBin;
}

cudaError_t order_blocks(const Params &p, int *blocks)
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, order_fn(p), kOrderBlock, 0);
    const long long need = (static_cast<long long>(p.npad) * kOrderLanes + kOrderBlock - 1) / kOrderBlock;
    const int most = per_sm * sms < kOrderMaxBlocks ? per_sm * sms : kOrderMaxBlocks;
    *blocks = static_cast<int>(need < most ? need : most);
    return e;
}

cudaError_t launch_order(const Params &p, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(p.order_blocks));
    cfg.blockDim = dim3(kOrderBlock);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {const_cast<Params *>(&p)};
    return cudaLaunchKernelExC(&cfg, order_fn(p), args);
}

} // namespace bsg
