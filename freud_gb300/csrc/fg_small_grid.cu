// The cell grid of one small system, and its query groups, in one block: counts, scan,
// scatter, ordering within cells and the group list from shared memory. The general build
// is two memsets and four to six launches, each a few microseconds of latency at these
// sizes: 1000 points 25 to 37 us of kernels, 11 to 12 here (8000: 22 to 28), launch included.
// Bound by latency: a chain of some ten block barriers and three trips to memory.
#include "fg_groups.cuh"
#include "fg_prof.cuh"

#include <algorithm>
#include <atomic>

namespace fg {

namespace {

constexpr int SG_T = 1024;

__device__ __forceinline__ uint32_t sort_size(uint32_t n)
{
    return n <= 64 ? 64u : 1u << (32 - __clz(n - 1));
}

// Ascending bitonic sort of n words in shared memory by the block, in its all-ascending form (a merge
// opens by comparing each element with its mirror): elements past n count as the largest. Neighbouring
// 32 pairs stay within 64 words while the pairs are at most 32 apart, so such stages need no
// barrier of the block.
__device__ __forceinline__ void block_sort(uint32_t* v, uint32_t n, uint32_t tid)
{
    const uint32_t np = sort_size(n);
    for (uint32_t k = 2; k <= np; k <<= 1)
    {
        for (uint32_t j = k >> 1; j > 0; j >>= 1)
        {
            const bool mirror = j == k >> 1;
            for (uint32_t p = tid; p < np / 2; p += SG_T)
            {
                const uint32_t in = p & (j - 1), first = 2 * (p - in);
                const uint32_t a = first + in, b = mirror ? first + k - 1 - in : a + j;
                if (b < n)
                {
                    const uint32_t x = v[a], y = v[b];
                    if (x > y)
                    {
                        v[a] = y;
                        v[b] = x;
                    }
                }
            }
            if (j > 32 || (j == 1 && k >= 64))
                __syncthreads();
            else
                __syncwarp();
        }
    }
}

// Points are put in order within their cells by counting, for each, those of smaller index in its
// cell, which takes the sum of the cells' squares; past SG_RANK_WORK times the sort's size the block sorts
// all of them by cell and index. 8192 points in one cell: ranks 430 to 1200 us, sorted 63; in 64
// cells 93 / 69; 5000 in 64 cells 30 / 48; 1000 in one 28 / 20.
constexpr uint32_t SG_RANK_WORK = 72;
static_assert(SMALL_N <= 1u << 13 && SMALL_CELLS <= 1u << 15, "a word holds cell and index");

__global__ void __launch_bounds__(SG_T)
    k_small_grid(SmallGrid a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_items;
    __shared__ uint32_t s_work; // sum of the squares of the cells' points
    const uint32_t ncell = a.F.ncell, n = a.n;
    uint32_t* const start = reinterpret_cast<uint32_t*>(smem_raw); // [ncell + 1] counts, then offsets
    uint32_t* const where = start + ncell + 1;                     // [n] cell | rank << 16, then slot
    uint32_t* const list = where + n;                              // [n] sorted: points by slot
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31;
    for (uint32_t c = tid; c <= ncell; c += SG_T)
        start[c] = 0;
    if (tid == 0)
        s_items = s_work = 0;
    __syncthreads();
    const int dim[3] = {a.F.dim[0], a.F.dim[1], a.F.dim[2]};
    int off = 0;
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += SG_T)
    {
        const float* p = a.pts + 3 * static_cast<size_t>(i);
        int cx, cy, cz, img;
        point_cell(a.F.b, dim, p[0], p[1], p[2], cx, cy, cz, img);
        const uint32_t cell = static_cast<uint32_t>(cx + dim[0] * (cy + dim[1] * cz));
        where[i] = cell | (atomicAdd(&start[cell], 1u) << 16);
        off |= img;
    }
    off = __syncthreads_or(off);
    if (a.out != nullptr && tid == 0)
        *a.out = off != 0;
    // exclusive scan of the counts: a run of cells a thread
    const uint32_t per = (ncell + SG_T - 1) / SG_T;
    const uint32_t c0 = min(ncell, tid * per), c1 = min(ncell, c0 + per);
    uint32_t sum = 0;
    for (uint32_t c = c0; c < c1; ++c)
        sum += start[c];
    uint32_t incl = warp_inclusive(sum, lane);
    if (lane == 31)
        s_warp[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32)
    {
        const uint32_t w = s_warp[lane];
        s_warp[lane] = warp_inclusive(w, lane) - w;
    }
    __syncthreads();
    uint32_t at = incl - sum + s_warp[tid >> 5], squares = 0;
    for (uint32_t c = c0; c < c1; ++c)
    {
        const uint32_t k = start[c];
        start[c] = at;
        at += k;
        squares += k * k;
    }
    if (tid == 0)
        start[ncell] = n;
    squares = __reduce_add_sync(GR_FULL, squares);
    if (lane == 0 && squares > 0)
        atomicAdd(&s_work, squares);
    __syncthreads();
    const bool full = a.sorted && s_work > SG_RANK_WORK * sort_size(n);
    for (uint32_t c = tid; c <= ncell; c += SG_T)
        a.start[c] = start[c];
    for (uint32_t i = tid; i < n; i += SG_T)
    {
        const uint32_t w = where[i];
        const uint32_t slot = start[w & 0xffffu] + (w >> 16);
        if (full)
            list[i] = ((w & 0xffffu) << 13) | i; // (below 2^15 cells, 2^13 points)
        else if (a.sorted)
            list[slot] = i;
        else
            where[i] = slot;
    }
    if (full)
    {
        __syncthreads();
        block_sort(list, n, tid);
        for (uint32_t s = tid; s < n; s += SG_T)
            where[list[s] & 8191u] = s;
        __syncthreads();
    }
    else if (a.sorted)
    {
        // a point's place in its cell: the points of smaller index
        __syncthreads();
        for (uint32_t i = tid; i < n; i += SG_T)
        {
            const uint32_t cell = where[i] & 0xffffu;
            const uint32_t s0 = start[cell], s1 = start[cell + 1];
            uint32_t slot = s0;
            for (uint32_t s = s0; s < s1; ++s)
                slot += list[s] < i ? 1u : 0u;
            where[i] = slot;
        }
    }
    // (each thread wrote the slots that it reads, or all waited)
#pragma unroll 4
    for (uint32_t i = tid; i < n; i += SG_T)
    {
        const float* p = a.pts + 3 * static_cast<size_t>(i);
        const float x = p[0], y = p[1], z = p[2];
        int img = 0;
        if (off != 0)
        {
            int cx, cy, cz;
            point_cell(a.F.b, dim, x, y, z, cx, cy, cz, img);
        }
        const uint32_t slot = where[i];
        a.cpos[slot] = make_float4(x, y, a.F.b.is2d ? 0.0f : z, __int_as_float(img));
        a.cidx[slot] = i;
    }
    if (a.items != nullptr)
    {
        for (uint32_t b0 = tid & ~31u; b0 < a.nboxes; b0 += SG_T)
        {
            const uint32_t b = b0 + lane;
            const uint32_t points = b < a.nboxes ? box_points(a.F, group_box(a.F, b), start) : 0u;
            append_groups(0, b, points, a.items, &s_items, lane);
        }
        __syncthreads();
        for (uint32_t w = tid; w < a.n_words; w += SG_T)
            a.words[w] = w == 0 ? s_items : 0u;
    }
}

} // namespace

size_t small_grid_smem(uint32_t n, uint32_t ncell, bool sorted)
{
    return sizeof(uint32_t) * (static_cast<size_t>(ncell) + 1 + static_cast<size_t>(n) * (sorted ? 2 : 1));
}

void launch_small_grid(const SmallGrid& a, cudaStream_t s)
{
    const size_t smem = small_grid_smem(a.n, a.F.ncell, a.sorted != 0);
    // more than 48 KB, static arrays included, has to be allowed: once a device, for the largest grid
    static std::atomic<uint64_t> allowed {0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = uint64_t(1) << (dev & 63);
    if (smem > 47 * 1024 && (allowed.load(std::memory_order_acquire) & bit) == 0)
    {
        cudaFuncSetAttribute(k_small_grid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(small_grid_smem(SMALL_N, SMALL_CELLS, true)));
        allowed.fetch_or(bit, std::memory_order_release);
    }
    ProfScope prof_("k_small_grid", s);
    k_small_grid<<<1, SG_T, smem, s>>>(a);
}

} // namespace fg
