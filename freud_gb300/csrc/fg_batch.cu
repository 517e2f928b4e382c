// Batched frames: every frame of a batch of uneven-N frames in one launch per
// stage.
//
// Grid build: one counting sort over the concatenated points, each point placed
// by its own frame's box (exact makeFractional, Box.h:243-255), so the cells of
// all frames form one array of offsets.
//
// Steinhardt neighbours: warp per cell over the 27-cell stencil (staged in
// shared memory, lanes over candidates), count then fill; the bonds of a frame
// batch feed the existing qlm / average / wl kernels over the concatenated
// rows, and the system sums are taken per frame.
#include "fg_groups.cuh"
#include "fg_prof.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

namespace fg {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Largest f with base[f] <= x (base[0] = 0 <= x < base[nframes]).
__device__ __forceinline__ uint32_t frame_of(const uint32_t* __restrict__ base, uint32_t nframes, uint32_t x)
{
    uint32_t lo = 0, hi = nframes;
    while (hi - lo > 1)
    {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(base + mid) <= x)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__global__ void k_frames_assign(const FrameDesc* __restrict__ fd, const uint32_t* __restrict__ pt_base,
                                uint32_t nframes, const float* __restrict__ pts, uint32_t n,
                                uint32_t* __restrict__ cell_of, uint32_t* __restrict__ rank, float4* __restrict__ pos4,
                                uint32_t* __restrict__ cell_count, int* __restrict__ frame_out)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const uint32_t fi = frame_of(pt_base, nframes, i);
        const FrameDesc& F = fd[fi];
        const float x = pts[3 * (size_t) i];
        const float y = pts[3 * (size_t) i + 1];
        const float z = pts[3 * (size_t) i + 2];
        const int dim[3] = {F.dim[0], F.dim[1], F.dim[2]};
        int cx, cy, cz, img;
        point_cell(F.b, dim, x, y, z, cx, cy, cz, img);
        const uint32_t cell = F.cell_base + static_cast<uint32_t>(cx + dim[0] * (cy + dim[1] * cz));
        cell_of[i] = cell;
        rank[i] = atomicAdd(&cell_count[cell], 1u);
        pos4[i] = make_float4(x, y, F.b.is2d ? 0.0f : z, __int_as_float(img));
        if (img != 0 && frame_out[fi] == 0)
            atomicOr(&frame_out[fi], 1);
    }
}

__global__ void k_frames_scatter(uint32_t n, const uint32_t* __restrict__ cell_of, const uint32_t* __restrict__ rank,
                                 const float4* __restrict__ pos4, const uint32_t* __restrict__ start,
                                 float4* __restrict__ cpos, uint32_t* __restrict__ cidx)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const uint32_t pos = start[cell_of[i]] + rank[i];
        cpos[pos] = pos4[i];
        if (cidx != nullptr)
            cidx[pos] = i;
    }
}

// Thread per box of cells: its points, split evenly over groups of at most 32.
__global__ void k_frames_groups(BatchGrid g, uint32_t nboxes, uint4* __restrict__ items, uint32_t* __restrict__ n_items)
{
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t f = 0, local = 0, n = 0;
    if (b < nboxes)
    {
        f = frame_of(g.box_base, g.nframes, b);
        const FrameDesc& F = g.fd[f];
        local = b - F.box_base;
        n = box_points(F, group_box(F, local), g.start);
    }
    append_groups(f, local, n, items, n_items, lane);
}

// ---------------------------------------------------------------------------
// Steinhardt neighbours (warp per cell, 27-cell stencil of r_max cells)
// ---------------------------------------------------------------------------
//
// A warp takes one home cell at a time (cells strided over the resident warps,
// ascending, so a warp meets each frame once). Its queries are the cell's own
// points, handled in groups of at most 32; for each group the stencil's
// candidates - item s in 0..26 (x fastest), slots in cell order: the fixed
// order in which each query's bonds are written and later summed - are staged in
// shared memory FB_TILE at a time, with the image vector that a query inside the
// box needs already resolved. For each query of the group the lanes test 32
// candidates per round (AABBQuery.cc:93,125 arithmetic); bonds keep candidate
// order. The count pass adds ballots; the fill pass appends each accepted bond
// (output row, p_j - q, r^2, j) to a per-warp queue that is drained 32 entries at
// a time, so the exact box.wrap of Steinhardt.cc:155 (three IEEE divisions) runs
// on full warps.

constexpr int FB_WARPS = 4;
constexpr int FB_THREADS = FB_WARPS * 32;
constexpr int FB_TILE = 128;  // staged candidates per warp
constexpr int FB_QUEUE = 64;  // bond queue entries per warp (drained at 32)
constexpr int FB_K0_OK = 1 << 24; // staged image resolved (query in the box)

template<bool FILL> struct FBWarp
{
    float4 pos[FB_TILE];      // x, y, z, point index (bits)
    float4 img[FB_TILE];      // image vector for a query in the box; w = packed n_j - wrap | FB_K0_OK
    float4 q[32];             // the group's queries (w = packed box image)
    uint32_t qi[32];
    unsigned long long qe[FILL ? FB_QUEUE : 1]; // fill: output row of a queued bond
    float4 qv[FILL ? FB_QUEUE : 1];             // fill: p_j - q (x, y, z), r^2
    uint32_t qj[FILL ? FB_QUEUE : 1];           // fill: neighbour index
    uint32_t it_off[28];      // stencil item offsets (prefix of counts)
    uint32_t it_start[27];    // first slot of the item's cell
    int it_wrap[27];          // (wx + 1) + 3 (wy + 1) + 9 (wz + 1)
};

// ONE (one pass, FILL): no counts and offsets beforehand. Each warp takes chunks of
// the bond arrays from a device counter (*alloc) and places each query's bonds at
// its chunk's cursor; before a query the chunk must hold the cell's candidate
// count, an upper bound on the query's bonds (else the rest of the chunk is left
// and a new one taken). seg[i] / counts[i] receive the query's first bond and its
// bond count. Bonds past cap are not written and a query whose bonds end past cap
// gets count 0 (the caller compares *alloc with cap and reruns the two passes when
// the arrays were too small; the kernels after this one never read past cap). A
// query's bonds keep candidate order, so the per-particle sums downstream are the
// same as with the two passes.
constexpr uint32_t FB_CHUNK = 4096; // bond slots a warp takes at a time (one pass)

// Cells of more than FB_HEAVY points would keep their warp busy long after the others are
// done: the first launch lists their queries in groups of FB_PART and the second (LISTED) takes those,
// a group a warp. W_l of 8192 points in one cell 1310 -> 13.6 ms, of a droplet of 8000 57 -> 4.9
// ms (groups of 32: 17 and 6.5).
constexpr uint32_t FB_HEAVY = 128;
constexpr uint32_t FB_PART = 8; // queries of a listed group

template<bool FILL, bool ONE, bool LISTED>
__global__ void __launch_bounds__(FB_THREADS, FILL ? 8 : 10)
    k_frames_ball(BatchGrid g, BallParams p, uint32_t* __restrict__ counts, const uint64_t* __restrict__ offsets,
                  uint32_t* __restrict__ bj, float4* __restrict__ bvd, uint32_t* __restrict__ seg,
                  unsigned long long* __restrict__ alloc, unsigned long long cap, uint2* __restrict__ heavy,
                  uint32_t* __restrict__ n_heavy)
{
    __shared__ FBWarp<FILL> sw[FB_WARPS];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    FBWarp<FILL>& W = sw[warp];
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t nwarps = gridDim.x * FB_WARPS;
    uint32_t at = blockIdx.x * FB_WARPS + warp; // cell, or item of the list
    const uint32_t work = LISTED ? *n_heavy : g.ncell;
    if (at >= work)
        return;
    uint32_t f = frame_of(g.cell_base, g.nframes, LISTED ? heavy[at].x : at);
    uint32_t qn = 0; // queued bonds (fill)
    unsigned long long cur = 0, cend = 0; // one pass: the warp's chunk [cur, cend)

    // drain the first n queued bonds: exact box.wrap of p_j - q in frame f
    auto drain = [&](uint32_t n) {
        if (lane < static_cast<int>(n))
        {
            const DevBox& B = g.fd[f].b;
            const unsigned long long e = W.qe[lane];
            const float4 v = W.qv[lane];
            float wx, wy, wz;
            box_wrap(B, v.x, v.y, v.z, wx, wy, wz);
            if (!ONE || e < cap)
            {
                bj[e] = W.qj[lane];
                bvd[e] = make_float4(wx, wy, wz, __fsqrt_rn(v.w));
            }
        }
        __syncwarp();
    };

    for (; at < work; at += nwarps)
    {
        const uint2 item = LISTED ? heavy[at] : make_uint2(at, 0u);
        const uint32_t c = item.x;
        const uint32_t q0 = g.start[c];
        const uint32_t nqc = LISTED ? min(g.start[c + 1] - q0, item.y + FB_PART) : g.start[c + 1] - q0;
        if (nqc == 0)
            continue;
        if (!LISTED && nqc > FB_HEAVY)
        {
            const uint32_t groups = (nqc + FB_PART - 1) / FB_PART;
            uint32_t to = 0;
            if (lane == 0)
                to = atomicAdd(n_heavy, groups);
            to = __shfl_sync(FULL, to, 0);
            for (uint32_t k = lane; k < groups; k += 32)
                heavy[to + k] = make_uint2(c, FB_PART * k);
            continue;
        }
        if (LISTED ? c < g.cell_base[f] || c >= g.cell_base[f + 1] : c >= g.cell_base[f + 1])
        {
            if (FILL && qn > 0)
            {
                drain(qn);
                qn = 0;
            }
            if (LISTED)
                f = frame_of(g.cell_base, g.nframes, c);
            while (c >= g.cell_base[f + 1])
                ++f;
        }
        const FrameDesc& F = g.fd[f];
        const int d0 = F.dim[0], d1 = F.dim[1], d2 = F.dim[2];
        const int lc = static_cast<int>(c - F.cell_base);
        const int cz = lc / (d0 * d1);
        const int cy = (lc / d0) % d1;
        const int cx = lc % d0;
        const int nst = F.b.is2d ? 9 : 27;
        // stencil items (lane s < nst), same enumeration as the reference order restated above
        {
            uint32_t cnt = 0, st = 0;
            int wr = 13;
            if (lane < nst)
            {
                const int ux = cx + lane % 3 - 1;
                const int uy = cy + (lane / 3) % 3 - 1;
                const int uz = cz + (F.b.is2d ? 0 : lane / 9 - 1);
                const int wx = ux < 0 ? -1 : (ux >= d0 ? 1 : 0);
                const int wy = uy < 0 ? -1 : (uy >= d1 ? 1 : 0);
                const int wz = uz < 0 ? -1 : (uz >= d2 ? 1 : 0);
                const uint32_t cell = F.cell_base +
                                      static_cast<uint32_t>((ux - wx * d0) + d0 * ((uy - wy * d1) + d1 * (uz - wz * d2)));
                st = g.start[cell];
                cnt = g.start[cell + 1] - st;
                wr = (wx + 1) + 3 * (wy + 1) + 9 * (wz + 1);
            }
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o)
                    incl += v;
            }
            if (lane < 27)
            {
                W.it_off[lane] = incl - cnt;
                W.it_start[lane] = st;
                W.it_wrap[lane] = wr;
            }
            if (lane == 26)
                W.it_off[27] = incl;
        }
        __syncwarp();
        const uint32_t T = W.it_off[27];
        const uint32_t ntile = (T + FB_TILE - 1) / FB_TILE;

        for (uint32_t g0 = item.y; g0 < nqc; g0 += 32)
        {
            const uint32_t ng = min(32u, nqc - g0);
            uint32_t my_cnt = 0;          // bonds so far of query g0 + lane
            uint64_t my_off = 0;
            if (lane < static_cast<int>(ng))
            {
                const uint32_t i = g.cidx[q0 + g0 + lane];
                W.q[lane] = g.cpos[q0 + g0 + lane];
                W.qi[lane] = i;
                if (FILL && !ONE)
                    my_off = offsets[i];
            }
            // one pass over the cell's tiles for the group: counts only (fill_now
            // false) or counts and bonds
            auto run_tiles = [&](bool fill_now, bool alloc_per_query) {
            for (uint32_t tile = 0; tile < ntile; ++tile)
            {
                const uint32_t t0 = tile * FB_TILE;
                const uint32_t TT = min(static_cast<uint32_t>(FB_TILE), T - t0);
                // stage candidates [t0, t0 + TT) unless this tile is already staged
                if (ntile > 1 || g0 == item.y)
                {
                    __syncwarp();
                    for (uint32_t tl = lane; tl < TT; tl += 32)
                    {
                        const uint32_t t = t0 + tl;
                        int s = 0;
#pragma unroll
                        for (int step = 16; step >= 1; step >>= 1)
                        {
                            if (s + step < 27 && W.it_off[s + step] <= t)
                                s += step;
                        }
                        const uint32_t slot = W.it_start[s] + (t - W.it_off[s]);
                        const float4 pp = g.cpos[slot];
                        const uint32_t j = g.cidx[slot];
                        const int wr = W.it_wrap[s];
                        const int pim = __float_as_int(pp.w);
                        const int kx = img_ax(pim, 0) - (wr % 3 - 1);
                        const int ky = img_ax(pim, 1) - ((wr / 3) % 3 - 1);
                        const int kz = img_ax(pim, 2) - (wr / 9 - 1);
                        int k0 = pack_image(kx, ky, kz);
                        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (kx >= -1 && kx <= 1 && ky >= -1 && ky <= 1 && kz >= -1 && kz <= 1)
                        {
                            const float* iv = F.b.img[(kx + 1) * 9 + (ky + 1) * 3 + (kz + 1)];
                            v.x = iv[0];
                            v.y = iv[1];
                            v.z = iv[2];
                            k0 |= FB_K0_OK;
                        }
                        v.w = __int_as_float(k0);
                        W.pos[tl] = make_float4(pp.x, pp.y, pp.z, __uint_as_float(j));
                        W.img[tl] = v;
                    }
                    __syncwarp();
                }
                for (uint32_t k = 0; k < ng; ++k)
                {
                    const float4 q = W.q[k];
                    const uint32_t qi = W.qi[k];
                    const int qimg = __float_as_int(q.w);
                    uint32_t base = __shfl_sync(FULL, my_cnt, k);
                    uint64_t off = FILL && !ONE ? __shfl_sync(FULL, my_off, k) : 0;
                    if (ONE && alloc_per_query)
                    {
                        // room for every candidate of the cell (bound on the bonds)
                        if (cend - cur < T)
                        {
                            const unsigned long long want = T > FB_CHUNK ? T : FB_CHUNK;
                            unsigned long long b0 = 0;
                            if (lane == 0)
                                b0 = atomicAdd(alloc, want);
                            cur = __shfl_sync(FULL, b0, 0);
                            cend = cur + want;
                        }
                        if (lane == static_cast<int>(k))
                            my_off = cur;
                    }
                    if (ONE)
                        off = __shfl_sync(FULL, my_off, k);
                    for (uint32_t r0 = 0; r0 < TT; r0 += 32)
                    {
                        const uint32_t tl = r0 + lane;
                        bool acc = false;
                        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
                        float rsq = 0.f;
                        if (tl < TT)
                        {
                            a = W.pos[tl];
                            const float4 v = W.img[tl];
                            const int k0 = __float_as_int(v.w);
                            float ix = v.x, iy = v.y, iz = v.z;
                            bool ok = (k0 & FB_K0_OK) != 0;
                            if (qimg != 0)
                            {
                                // query outside the box: image k = n_j - n_q - wrap
                                const int kx = img_ax(k0, 0) - img_ax(qimg, 0);
                                const int ky = img_ax(k0, 1) - img_ax(qimg, 1);
                                const int kz = img_ax(k0, 2) - img_ax(qimg, 2);
                                ok = kx >= -1 && kx <= 1 && ky >= -1 && ky <= 1 && kz >= -1 && kz <= 1;
                                if (ok)
                                {
                                    const float* iv = F.b.img[(kx + 1) * 9 + (ky + 1) * 3 + (kz + 1)];
                                    ix = iv[0];
                                    iy = iv[1];
                                    iz = iv[2];
                                }
                            }
                            if (ok && !(p.exclude_ii && __float_as_uint(a.w) == qi))
                            {
                                const float rx = __fsub_rn(a.x, __fadd_rn(q.x, ix));
                                const float ry = __fsub_rn(a.y, __fadd_rn(q.y, iy));
                                const float rz = __fsub_rn(a.z, __fadd_rn(q.z, iz));
                                rsq = dot3(rx, ry, rz);
                                acc = rsq < p.r_max_sq && rsq >= p.r_min_sq;
                            }
                        }
                        const unsigned bal = __ballot_sync(FULL, acc);
                        if (FILL && fill_now && bal != 0)
                        {
                            if (acc)
                            {
                                const uint32_t slot = qn + __popc(bal & lt);
                                W.qe[slot] = off + base + __popc(bal & lt);
                                W.qv[slot] = make_float4(__fsub_rn(a.x, q.x), __fsub_rn(a.y, q.y),
                                                         __fsub_rn(a.z, q.z), rsq);
                                W.qj[slot] = __float_as_uint(a.w);
                            }
                            qn += __popc(bal);
                            __syncwarp();
                            if (qn >= 32)
                            {
                                drain(32);
                                const uint32_t rest = qn - 32;
                                unsigned long long e = 0;
                                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                                uint32_t j = 0;
                                if (lane < static_cast<int>(rest))
                                {
                                    e = W.qe[32 + lane];
                                    v = W.qv[32 + lane];
                                    j = W.qj[32 + lane];
                                }
                                __syncwarp();
                                if (lane < static_cast<int>(rest))
                                {
                                    W.qe[lane] = e;
                                    W.qv[lane] = v;
                                    W.qj[lane] = j;
                                }
                                __syncwarp();
                                qn = rest;
                            }
                        }
                        base += __popc(bal);
                    }
                    if (lane == static_cast<int>(k))
                        my_cnt = base;
                    if (ONE && alloc_per_query)
                        cur += base; // the query's bonds are placed: advance the cursor
                }
            }
            };
            if (!ONE)
            {
                run_tiles(FILL, false);
            }
            else if (ntile == 1)
            {
                // every candidate in one tile: each query's bonds are found in one
                // sweep, placed at the cursor with room for all candidates
                run_tiles(true, true);
            }
            else
            {
                // several tiles: count the group's bonds, place the group, then fill
                run_tiles(false, false);
                uint32_t incl = lane < static_cast<int>(ng) ? my_cnt : 0u;
                const uint32_t mine = incl;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const uint32_t v = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o)
                        incl += v;
                }
                const unsigned long long tot = __shfl_sync(FULL, incl, 31);
                if (cend - cur < tot)
                {
                    const unsigned long long want = tot > FB_CHUNK ? tot : FB_CHUNK;
                    unsigned long long b0 = 0;
                    if (lane == 0)
                        b0 = atomicAdd(alloc, want);
                    cur = __shfl_sync(FULL, b0, 0);
                    cend = cur + want;
                }
                my_off = cur + (incl - mine);
                cur += tot;
                my_cnt = 0;
                run_tiles(true, false);
            }
            if ((!FILL || ONE) && lane < static_cast<int>(ng))
            {
                // one pass: a query whose bonds do not fit below cap gets no bonds,
                // so the kernels after this one read nothing past the arrays (the
                // caller reruns the two passes)
                const bool fits = !ONE || my_off + my_cnt <= cap;
                counts[W.qi[lane]] = fits ? my_cnt : 0u;
                if (ONE)
                    seg[W.qi[lane]] = fits ? static_cast<uint32_t>(my_off) : 0u;
            }
            __syncwarp();
        }
    }
    if (FILL && qn > 0)
        drain(qn);
}

__global__ void __launch_bounds__(256) k_fullest_cell(BatchGrid g, uint32_t* __restrict__ most)
{
    uint32_t m = 0;
    for (uint32_t c = blockIdx.x * 256 + threadIdx.x; c < g.ncell; c += gridDim.x * 256)
        m = max(m, g.start[c + 1] - g.start[c]);
    m = __reduce_max_sync(FULL, m);
    if ((threadIdx.x & 31) == 0 && m > 0)
        atomicMax(most, m);
}

// ---------------------------------------------------------------------------
// Per-frame system sums
// ---------------------------------------------------------------------------

// hi + lo += v with the rounding error of hi + v kept exactly (TwoSum).
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float v)
{
    const float s = __fadd_rn(hi, v);
    const float bp = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(v, bp));
    hi = s;
    lo = __fadd_rn(lo, err);
}

// Rows [r0, r1) of one frame split. For each l, the (row, m) block of qlm is read
// with consecutive threads on consecutive values (thread t: column t mod (2l+1),
// row offset t div (2l+1), rows advancing by 256 div (2l+1)): coalesced loads. Each
// thread keeps float-float running sums (hi + lo, every addition an exact two-sum,
// Knuth's TwoSum: about 48 significant bits, far below the float32 inputs' own
// rounding, on the FP32 pipe instead of GB300's slow FP64 one); the threads of a
// column are then added in FP64 in a fixed order through shared memory and
// partial[f][split][col] is written (the same order every run). A block takes one l
// (blockIdx.z): a thread's sums are a serial chain, and one row at a time, all l in turn,
// left the chip waiting for loads (256k particles, l = 4, 6, .., 12, 174 MB:
// 0.105 ms, now 0.041).
constexpr int SYS_AHEAD = 8;
__global__ void __launch_bounds__(256)
    k_frames_sys(const uint32_t* __restrict__ pt_base, StLs ls, int stride, int splits,
                 const float2* __restrict__ src, double* __restrict__ partial)
{
    __shared__ double s_re[256];
    __shared__ double s_im[256];
    const uint32_t f = blockIdx.x;
    const uint32_t split = blockIdx.y;
    const uint32_t r_lo = pt_base[f];
    const uint32_t nf = pt_base[f + 1] - r_lo;
    const uint32_t per = (nf + splits - 1) / splits;
    const uint32_t r0 = r_lo + min(nf, split * per);
    const uint32_t r1 = r_lo + min(nf, (split + 1) * per);
    const int t = threadIdx.x;
    const int k = blockIdx.z;
    int col0 = 0;
    for (int q = 0; q < k; ++q)
        col0 += 2 * ls.l[q] + 1;
    const int nm = 2 * ls.l[k] + 1;
    const int rows_per_pass = blockDim.x / nm;
    const int m = t % nm;
    const int rr = t / nm;
    float hr = 0.f, lr = 0.f, hi = 0.f, li = 0.f;
    if (rr < rows_per_pass)
    {
        // SYS_AHEAD rows in flight; a missing one adds +0, which changes nothing
        const float2* base = src + ls.qlm_offset[k] + m;
        for (uint32_t r = r0 + rr; r < r1; r += SYS_AHEAD * rows_per_pass)
        {
            float2 v[SYS_AHEAD];
#pragma unroll
            for (int u = 0; u < SYS_AHEAD; ++u)
            {
                const uint32_t ru = r + u * rows_per_pass;
                v[u] = ru < r1 ? base[static_cast<size_t>(ru) * nm] : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < SYS_AHEAD; ++u)
            {
                two_sum_acc(hr, lr, v[u].x);
                two_sum_acc(hi, li, v[u].y);
            }
        }
    }
    s_re[t] = static_cast<double>(hr) + static_cast<double>(lr);
    s_im[t] = static_cast<double>(hi) + static_cast<double>(li);
    __syncthreads();
    if (t < nm)
    {
        double ar = 0.0, ai = 0.0;
        for (int q = 0; q < rows_per_pass; ++q)
        {
            ar += s_re[q * nm + t];
            ai += s_im[q * nm + t];
        }
        double* out = partial + ((static_cast<size_t>(f) * splits + split) * stride + col0 + t) * 2;
        out[0] = ar;
        out[1] = ai;
    }
}

// Blocks of 8 columns per frame, warp per column: the split sums reduced by lanes
// (every 32nd split) and a fixed shuffle tree (the same order every run), divided
// by n_f.
__global__ void __launch_bounds__(256)
    k_frames_sys_final(const uint32_t* __restrict__ pt_base, int stride, int splits,
                       const double* __restrict__ partial, double* __restrict__ sys)
{
    const uint32_t f = blockIdx.x;
    const int lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    const double nf = static_cast<double>(pt_base[f + 1] - pt_base[f]);
    for (int col = blockIdx.y * warps + (threadIdx.x >> 5); col < stride; col += warps * gridDim.y)
    {
        double sr = 0.0, si = 0.0;
        for (int k = lane; k < splits; k += 32)
        {
            const double* v = partial + ((static_cast<size_t>(f) * splits + k) * stride + col) * 2;
            sr += v[0];
            si += v[1];
        }
        for (int o = 16; o > 0; o >>= 1)
        {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            si += __shfl_xor_sync(0xffffffffu, si, o);
        }
        if (lane == 0)
        {
            sys[2 * (static_cast<size_t>(f) * stride + col)] = nf > 0.0 ? sr / nf : 0.0;
            sys[2 * (static_cast<size_t>(f) * stride + col) + 1] = nf > 0.0 ? si / nf : 0.0;
        }
    }
}

int grid_blocks(size_t n, int threads)
{
    size_t b = (n + threads - 1) / threads;
    if (b > 152 * 32)
        b = 152 * 32;
    return b < 1 ? 1 : static_cast<int>(b);
}

int sms()
{
    static int v = 0;
    if (v == 0)
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        if (v <= 0)
            v = 1;
    }
    return v;
}

} // namespace

void launch_frames_assign(const FrameDesc* fd, const uint32_t* pt_base, uint32_t nframes, const float* pts, uint32_t n,
                          uint32_t* cell_of, uint32_t* rank, float4* pos4, uint32_t* cell_count, int* frame_out,
                          cudaStream_t s)
{
    if (n == 0)
        return;
    ProfScope prof_("k_frames_assign", s);
    k_frames_assign<<<grid_blocks(n, 256), 256, 0, s>>>(fd, pt_base, nframes, pts, n, cell_of, rank, pos4, cell_count,
                                                         frame_out);
}

void launch_frames_groups(const BatchGrid& g, uint32_t nboxes, uint4* items, uint32_t* n_items, cudaStream_t s)
{
    if (nboxes == 0)
        return;
    ProfScope prof_("k_frames_groups", s);
    k_frames_groups<<<(nboxes + 127) / 128, 128, 0, s>>>(g, nboxes, items, n_items);
}

// Expected groups of a box whose point count is Poisson with the given mean.
static double expected_groups(double mean)
{
    static const std::vector<double> table = [] {
        std::vector<double> t(129, 0.0);
        for (int q = 1; q <= 128; ++q)
        {
            double p = std::exp(-static_cast<double>(q)), e = 0.0;
            for (int x = 1; x <= 4 * 128; ++x)
            {
                p *= static_cast<double>(q) / x;
                e += p * ((x + 31) / 32);
            }
            t[q] = e;
        }
        return t;
    }();
    if (mean >= 128.0)
        return mean / 32.0 + 0.5;
    const int i = static_cast<int>(mean);
    const double w = mean - i;
    return table[i] * (1.0 - w) + table[i + 1] * w;
}

// The box of cells that minimises cost(groups a box, cells met by a group, those of its own
// row of boxes, points a box) for uniform points. A box has at most 32 rows of
// cells (a lane each). Returns how many groups there are; cost < 0 leaves a shape out.
// r: the stencil's reach in cells. *cells_met: of a group of the best shape.
template<typename C>
static double best_boxes(const int dim[3], uint32_t n, double r, int nb[3], C cost, double* cells_met = nullptr)
{
    const double m = static_cast<double>(n) / (static_cast<double>(dim[0]) * dim[1] * dim[2]);
    const bool flat = dim[2] == 1;
    double best = 0.0, count = n;
    for (int a = 0; a < 3; ++a)
        nb[a] = dim[a];
    for (int kz = 1; kz <= (flat ? 1 : 6); ++kz)
    {
        for (int ky = 1; ky <= 6; ++ky)
        {
            for (int kx = 1; kx <= 8; ++kx)
            {
                const int k[3] = {kx, ky, kz};
                int b[3], top[3];
                double side[3];
                for (int a = 0; a < 3; ++a)
                {
                    b[a] = std::max(1, (dim[a] + k[a] - 1) / k[a]);
                    top[a] = (dim[a] + b[a] - 1) / b[a];
                    side[a] = static_cast<double>(dim[a]) / b[a];
                }
                if (top[1] * top[2] > 32)
                    continue;
                const double q = m * side[0] * side[1] * side[2];
                const double groups = expected_groups(q);
                if (groups <= 0.0)
                    continue;
                double v, row; // a group's stencil and its box row's part of it
                if (flat)
                {
                    const double sy = side[1] / std::max(1.0, q / 32.0);
                    v = side[0] * sy + 2.0 * r * (side[0] + sy) + M_PI * r * r;
                    row = side[1] * (side[0] + 2.0 * r);
                }
                else
                {
                    const double sz = side[2] / std::max(1.0, q / 32.0);
                    v = side[0] * side[1] * sz + 2.0 * r * (side[0] * side[1] + side[1] * sz + sz * side[0]) +
                        M_PI * r * r * (side[0] + side[1] + sz) + 4.0 / 3.0 * M_PI * r * r * r;
                    row = side[1] * side[2] * (side[0] + 2.0 * r);
                }
                const double c = cost(groups, v, row, q);
                if (c >= 0.0 && (best == 0.0 || c < best))
                {
                    best = c;
                    if (cells_met != nullptr)
                        *cells_met = v;
                    count = groups * b[0] * b[1] * b[2];
                    for (int a = 0; a < 3; ++a)
                        nb[a] = b[a];
                }
            }
        }
    }
    return count;
}

// The box minimising the work per point of uniform points: groups a box times (the
// candidates met, about 20 warp instructions each, plus about 600 of set-up), over the
// points of a box. Met is half the stencil of a group's bounds, and of its own row of
// boxes most. (64 uneven frames, r_max 4, cells of 2: boxes of 2 x 2 x 1 cells 11.9 ms,
// 2 x 2 x 5 12.5, 4 x 4 x 2 14.4, single cells 23.0.)
double group_boxes(const int dim[3], uint32_t n, int shell, int nb[3])
{
    const double m = static_cast<double>(n) / (static_cast<double>(dim[0]) * dim[1] * dim[2]);
    return best_boxes(dim, n, shell, nb, [m](double groups, double v, double row, double q) {
        return groups * (10.0 * (v + row) * m + 600.0) / q;
    });
}

// The same for the NeighborList passes, np points met by groups of the nq queries: about 8 warp
// instructions a candidate (the sweep), 1500 a group, and its sort by the room that the
// candidates need (8, 16 or 32 words a lane: 700, 1700, 4500). A shape just inside the next
// smaller room is worth fewer queries a group: 200k points, r_max 2.7, count 0.121 ms against
// 0.169 by a cost without the steps; a crystal of 256k, r_max 2.6, 0.138 / 0.181. *met:
// candidates of a group; shapes of more than 900 or of more than one full group are left out
// (0 if all are).
double nl_boxes(const int dim[3], uint32_t nq, uint32_t np, double reach, int nb[3], double* met)
{
    const double m = static_cast<double>(np) / (static_cast<double>(dim[0]) * dim[1] * dim[2]);
    double cells = 0.0;
    const double count = best_boxes(
        dim, nq, reach, nb,
        [m](double groups, double v, double, double q) {
            const double t = v * m, most = t + 5.0 * std::sqrt(t);
            const double fixed = most <= 256.0 ? 2200.0 : (most <= 512.0 ? 3200.0 : 6000.0);
            return t > 900.0 || q > 30.0 ? -1.0 : groups * (8.0 * t + fixed) / q;
        },
        &cells);
    *met = cells * m;
    return count;
}

void launch_frames_scatter(uint32_t n, const uint32_t* cell_of, const uint32_t* rank, const float4* pos4,
                           const uint32_t* start, float4* cpos, uint32_t* cidx, cudaStream_t s)
{
    if (n == 0)
        return;
    ProfScope prof_("k_frames_scatter", s);
    k_frames_scatter<<<grid_blocks(n, 256), 256, 0, s>>>(n, cell_of, rank, pos4, start, cpos, cidx);
}

namespace {
// one wave of resident blocks, or fewer when the grid has few cells
template<typename K> uint32_t frames_ball_blocks(K kernel, uint32_t ncell)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, FB_THREADS, 0);
    const uint32_t want = static_cast<uint32_t>(sms()) * static_cast<uint32_t>(std::max(per_sm, 1));
    return std::max(1u, std::min<uint32_t>(want, (ncell + FB_WARPS - 1) / FB_WARPS));
}
} // namespace

namespace {
// The cells and then the groups of the heavy ones.
template<bool FILL, bool ONE>
void frames_ball(const char* name, const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                 uint32_t* counts, const uint64_t* offsets, uint32_t* bond_j, float4* bond_vd, uint32_t* seg,
                 unsigned long long* alloc, uint64_t cap, cudaStream_t s)
{
    if (n == 0 || g.ncell == 0)
        return;
    cudaMemsetAsync(heavy.n, 0, sizeof(uint32_t), s);
    auto go = [&](auto kernel, const char* what, uint32_t items) {
        ProfScope prof_(what, s);
        kernel<<<frames_ball_blocks(kernel, items), FB_THREADS, 0, s>>>(g, p, counts, offsets, bond_j, bond_vd, seg, alloc,
                                                                      cap, heavy.items, heavy.n);
    };
    go(k_frames_ball<FILL, ONE, false>, name, g.ncell);
    if (n > FB_HEAVY)
        go(k_frames_ball<FILL, ONE, true>, "k_frames_ball<LISTED>", static_cast<uint32_t>(ball_heavy_items(n)));
}
} // namespace

void launch_fullest_cell(const BatchGrid& g, uint32_t* most, cudaStream_t s)
{
    ProfScope prof_("k_fullest_cell", s);
    k_fullest_cell<<<grid_blocks(g.ncell, 256 * 4), 256, 0, s>>>(g, most);
}

size_t ball_heavy_items(uint32_t n)
{
    return n / FB_PART + n / FB_HEAVY + 1;
}

void launch_frames_ball_count(const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                              uint32_t* counts, cudaStream_t s)
{
    frames_ball<false, false>("k_frames_ball<COUNT>", g, p, n, heavy, counts, nullptr, nullptr, nullptr, nullptr, nullptr,
                              0, s);
}

void launch_frames_ball_fill(const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                             const uint64_t* offsets, uint32_t* bond_j, float4* bond_vd, cudaStream_t s)
{
    frames_ball<true, false>("k_frames_ball<FILL>", g, p, n, heavy, nullptr, offsets, bond_j, bond_vd, nullptr, nullptr, 0,
                             s);
}

uint64_t frames_ball_onepass_slack(uint32_t ncell, uint32_t n)
{
    // every warp of either launch may leave the rest of its last chunk unused
    const uint64_t blocks = frames_ball_blocks(k_frames_ball<true, true, false>, ncell) +
        (n > FB_HEAVY ? frames_ball_blocks(k_frames_ball<true, true, true>, static_cast<uint32_t>(ball_heavy_items(n))) : 0u);
    return blocks * FB_WARPS * FB_CHUNK;
}

void launch_frames_ball_onepass(const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                                uint32_t* counts, uint32_t* seg, uint32_t* bond_j, float4* bond_vd,
                                unsigned long long* alloc, uint64_t cap, cudaStream_t s)
{
    frames_ball<true, true>("k_frames_ball<ONE>", g, p, n, heavy, counts, nullptr, bond_j, bond_vd, seg, alloc, cap, s);
}

int frames_sys_splits(uint32_t max_rows)
{
    const uint32_t want = (max_rows + FRAME_SYS_ROWS - 1) / FRAME_SYS_ROWS;
    return static_cast<int>(std::min<uint32_t>(std::max<uint32_t>(want, 1u), 65535u));
}

void launch_frames_sys(const uint32_t* pt_base, uint32_t nframes, uint32_t max_rows, const StLs& ls, int stride,
                       const float2* src, double* partial, double* sys, cudaStream_t s)
{
    if (nframes == 0)
        return;
    const int splits = frames_sys_splits(max_rows);
    {
        ProfScope prof_("k_frames_sys", s);
        k_frames_sys<<<dim3(nframes, splits, ls.nl), 256, 0, s>>>(pt_base, ls, stride, splits, src, partial);
    }
    launch_frames_sys_final(pt_base, nframes, max_rows, stride, partial, sys, s);
}

void launch_frames_sys_final(const uint32_t* pt_base, uint32_t nframes, uint32_t max_rows, int stride,
                             const double* partial, double* sys, cudaStream_t s)
{
    ProfScope prof_("k_frames_sys_final", s);
    k_frames_sys_final<<<dim3(nframes, (stride + 7) / 8), 256, 0, s>>>(pt_base, stride, frames_sys_splits(max_rows),
                                                                     partial, sys);
}

} // namespace fg
