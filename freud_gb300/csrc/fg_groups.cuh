// Query groups: the unit of work of the batched ball kernels (histogram,
// Steinhardt). Each frame's cells are tiled by boxes of cells (FrameDesc::nb boxes
// per axis, sized for about 30 points); a group is at most 32 points of one box,
// one per lane of a warp. A warp holds its group's positions in registers and
// streams the candidates of the group's stencil past them: lanes load 32
// candidates at a time, drop those farther than r_max from the bounds of the
// group, place the rest in a per-warp buffer, and every lane then meets each
// buffered candidate (a broadcast shared load) - no block barriers, no per-pair
// ballot, and one exact test per (group, kept candidate).
//
// Why groups and not a block per cell: a block had to meet at eight barriers per
// cell and to build its candidate lists with every warp, which took most of the
// histogram's time (64 uneven frames of 18.3 M points, r_max 4, density 0.85: of
// 16.9 ms, 1.6 ms were the shared adds and next to nothing the square roots).
#pragma once

#include "fg_batch.cuh"
#include "fg_packed.cuh"

namespace fg {
namespace {

constexpr unsigned GR_FULL = 0xffffffffu;
constexpr int GR_BUF = 64; // buffered candidates per warp and kind (32 pending + one round)

constexpr float GR_FAR = -3e30f; // padding of a candidate buffer: every r^2 with it is infinite

__device__ __forceinline__ float redux_min(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ float redux_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t u = __shfl_up_sync(GR_FULL, v, o);
        if (lane >= o)
            v += u;
    }
    return v;
}

// Largest s with off(lane s) <= t, off ascending over the lanes, off(lane 0) = 0.
__device__ __forceinline__ int warp_run_of(uint32_t off, uint32_t t)
{
    int s = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1)
    {
        const uint32_t o = __shfl_sync(GR_FULL, off, s + step);
        if (o <= t)
            s += step;
    }
    return s;
}

// Cells [lo, hi) of box index b of n boxes over d cells.
__device__ __forceinline__ int box_edge(int b, int d, int n)
{
    return static_cast<int>(static_cast<uint32_t>(b) * static_cast<uint32_t>(d) / static_cast<uint32_t>(n));
}

struct GroupBox
{
    int lo[3], hi[3]; // cells of the group's box, per axis
    int b[3];         // its index
};

__device__ __forceinline__ GroupBox group_box(const FrameDesc& F, uint32_t local)
{
    const uint32_t n0 = F.nb[0], n1 = F.nb[1];
    GroupBox g;
    g.b[0] = static_cast<int>(local % n0);
    g.b[1] = static_cast<int>(local / n0 % n1);
    g.b[2] = static_cast<int>(local / n0 / n1);
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        g.lo[a] = box_edge(g.b[a], F.dim[a], F.nb[a]);
        g.hi[a] = box_edge(g.b[a] + 1, F.dim[a], F.nb[a]);
    }
    return g;
}

// Points in a box of cells.
__device__ __forceinline__ uint32_t box_points(const FrameDesc& F, const GroupBox& gb, const uint32_t* __restrict__ start)
{
    uint32_t n = 0;
    for (int z = gb.lo[2]; z < gb.hi[2]; ++z)
    {
        for (int y = gb.lo[1]; y < gb.hi[1]; ++y)
        {
            const uint32_t row = F.cell_base + static_cast<uint32_t>(F.dim[0] * (y + F.dim[1] * z));
            n += start[row + gb.hi[0]] - start[row + gb.lo[0]];
        }
    }
    return n;
}

// Appends the groups of this lane's box (frame f, box local, n points) to the list; every
// lane of the warp calls it.
__device__ __forceinline__ void append_groups(uint32_t f, uint32_t local, uint32_t n, uint4* __restrict__ items,
                                              uint32_t* __restrict__ n_items, int lane)
{
    const uint32_t groups = (n + 31) / 32;
    const uint32_t incl = warp_inclusive(groups, lane);
    uint32_t base = 0;
    if (lane == 31 && incl > 0)
        base = atomicAdd(n_items, incl);
    base = __shfl_sync(GR_FULL, base, 31) + incl - groups;
    for (uint32_t k = 0; k < groups; ++k)
    {
        const uint32_t q0 = static_cast<uint32_t>(static_cast<uint64_t>(n) * k / groups);
        const uint32_t q1 = static_cast<uint32_t>(static_cast<uint64_t>(n) * (k + 1) / groups);
        items[base + k] = make_uint4(f, local, q0, q1 - q0);
    }
}

// Slot of the lane's query: query first + lane of the box's points in cell order
// (rows of x-cells are contiguous slot runs, at most 32 rows a box).
__device__ __forceinline__ uint32_t group_slot(const FrameDesc& F, const GroupBox& gb, const uint32_t* __restrict__ start,
                                               uint32_t first, int lane)
{
    const int ny = gb.hi[1] - gb.lo[1], nz = gb.hi[2] - gb.lo[2];
    const int z = gb.lo[2] + lane / ny;
    uint32_t st = 0, cnt = 0;
    if (lane < ny * nz)
    {
        const int y = gb.lo[1] + lane % ny;
        const uint32_t row = F.cell_base + static_cast<uint32_t>(F.dim[0] * (y + F.dim[1] * z));
        st = start[row + gb.lo[0]];
        cnt = start[row + gb.hi[0]] - st;
    }
    const uint32_t off = warp_inclusive(cnt, lane) - cnt;
    const uint32_t t = first + static_cast<uint32_t>(lane);
    const int r = warp_run_of(off, t);
    return __shfl_sync(GR_FULL, st - off, r) + t;
}

// What bounds a group's candidates.
struct GroupBounds
{
    float lo[3], hi[3]; // of the group's positions
    float cull, cull2;  // radius (and its square) beyond which candidates are dropped
    bool clip;          // rows and x-cells of the stencil beyond the cull radius of the
                        // bounds are left out (every point in the box, box without tilt)
    bool half;          // half stencil, see stencil_runs
    uint32_t after;     // half: the group's first slot
};

// Squared distance of a point from the bounds.
__device__ __forceinline__ float group_gap2(const GroupBounds& gd, float x, float y, float z)
{
    const float gx = fmaxf(fmaxf(gd.lo[0] - x, x - gd.hi[0]), 0.f);
    const float gy = fmaxf(fmaxf(gd.lo[1] - y, y - gd.hi[1]), 0.f);
    const float gz = fmaxf(fmaxf(gd.lo[2] - z, z - gd.hi[2]), 0.f);
    return gx * gx + gy * gy + gz * gz;
}

// The rows (y, z) of cells of a group's stencil, unwrapped: those of the group's box
// widened by the shell, or, with clip, those of them within the cull radius of the
// bounds along y and along z.
struct StencilRows
{
    int y0, ny, z0, n;
    int segs; // runs a row: 1 when no x-cell of it lies across the boundary, else 3
};

// Cell of a bound, far from the integers' ends: bounds are infinite where a coordinate is.
__device__ __forceinline__ int bound_cell(float v)
{
    return static_cast<int>(floorf(fminf(fmaxf(v, -1e6f), 1e6f)));
}

// (wide: half-width in place of the frame's shell.)
__device__ __forceinline__ StencilRows stencil_rows(const FrameDesc& F, const GroupBox& gb, const GroupBounds& gd,
                                                    int wide = 0)
{
    const int s = wide > 0 ? wide : F.shell;
    const bool flat = F.b.is2d != 0;
    int ya = gb.lo[1] - s, yb = gb.hi[1] + s;
    int za = flat ? 0 : gb.lo[2] - s, zb = flat ? 1 : gb.hi[2] + s;
    if (gd.clip)
    {
        // cell edges carry the rounding of the fractional coordinates (1e-3 of a cell is
        // far above it)
        const float r = gd.cull;
        ya = max(ya, bound_cell((gd.lo[1] - r - F.b.lo[1]) * F.cells_per[1] - 1e-3f));
        yb = min(yb, bound_cell((gd.hi[1] + r - F.b.lo[1]) * F.cells_per[1] + 1e-3f) + 1);
        if (!flat)
        {
            za = max(za, bound_cell((gd.lo[2] - r - F.b.lo[2]) * F.cells_per[2] - 1e-3f));
            zb = min(zb, bound_cell((gd.hi[2] + r - F.b.lo[2]) * F.cells_per[2] + 1e-3f) + 1);
        }
    }
    StencilRows R;
    R.y0 = ya;
    R.ny = max(yb - ya, 0); // (none around an infinite coordinate)
    R.z0 = za;
    R.n = R.ny * max(zb - za, 0);
    R.segs = gb.lo[0] >= s && gb.hi[0] + s <= F.dim[0] ? 1 : 3;
    return R;
}

constexpr int RUN_OWN = 32; // run of the group's own row of boxes (half stencil)

// A chunk of a group's stencil as runs of consecutive slots, one per lane.
struct StencilRuns
{
    uint32_t first; // this lane's first slot - off
    uint32_t off;   // candidates before this lane's run
    int wrap;       // (wx + 1) + 3 (wy + 1) + 9 (wz + 1), | RUN_OWN
    uint32_t total; // candidates of the chunk
    bool plain;     // every run has wrap 13 (none across the boundary)
};

__device__ __forceinline__ int rows_per_chunk(const StencilRows& R)
{
    return R.segs == 1 ? 32 : 10;
}

// The runs of rows [row0, row0 + rows_per_chunk).
//
// half: each unordered pair of image 0 is met from one of its ends only. Rows of cells
// belong to rows of boxes (box indices along y and z); two groups in different rows of
// boxes meet from the end that the parity of the indices' sum picks - about half of the
// rows around a group, whole - and inside one row of boxes from the end of the smaller
// slot (slots up to the group's first are left out here, the kernel tests the rest).
// Order by slot alone would leave out
// only what lies before the group's first plane: 0.65 of the stencil of a group 2 deep
// (r_max 4) instead of 0.5.
__device__ __forceinline__ StencilRuns stencil_runs(const FrameDesc& F, const GroupBox& gb, const StencilRows& R,
                                                    const uint32_t* __restrict__ start, int row0, const GroupBounds& gd,
                                                    int lane, int wide = 0)
{
    const int d0 = F.dim[0], d1 = F.dim[1], d2 = F.dim[2];
    const int s = wide > 0 ? wide : F.shell;
    const int rr = row0 + (R.segs == 1 ? lane : lane / 3);
    const int k = R.segs == 1 ? 1 : lane % 3;
    uint32_t st = 0, cnt = 0;
    int wrap = 13;
    if (rr < R.n && (R.segs == 1 || lane < 30))
    {
        const int zi = rr / R.ny;
        const int uy = R.y0 + (rr - zi * R.ny), uz = R.z0 + zi;
        const int wz = uz < 0 ? -1 : (uz >= d2 ? 1 : 0);
        const int wy = uy < 0 ? -1 : (uy >= d1 ? 1 : 0);
        int xa = gb.lo[0] - s, xb = gb.hi[0] - 1 + s;
        if (gd.clip)
        {
            const float cy = F.cell_width[1];
            const float ya = F.b.lo[1] + (uy - 1e-3f) * cy, yb = F.b.lo[1] + (uy + 1.001f) * cy;
            const float gy = fmaxf(fmaxf(ya - gd.hi[1], gd.lo[1] - yb), 0.0f);
            float g2 = gy * gy;
            if (!F.b.is2d)
            {
                const float cz = F.cell_width[2];
                const float za = F.b.lo[2] + (uz - 1e-3f) * cz, zb = F.b.lo[2] + (uz + 1.001f) * cz;
                const float gz = fmaxf(fmaxf(za - gd.hi[2], gd.lo[2] - zb), 0.0f);
                g2 += gz * gz;
            }
            if (g2 > gd.cull2)
            {
                xb = xa - 1;
            }
            else
            {
                const float r = sqrtf(gd.cull2 - g2);
                xa = max(xa, bound_cell((gd.lo[0] - r - F.b.lo[0]) * F.cells_per[0] - 1e-3f));
                xb = min(xb, bound_cell((gd.hi[0] + r - F.b.lo[0]) * F.cells_per[0] + 1e-3f));
            }
        }
        bool mine = true, own_row = false;
        if (gd.half && wy == 0 && wz == 0)
        {
            // box indices: the largest with box_edge <= the cell
            const int by = ((uy + 1) * F.nb[1] - 1) / d1, bz = ((uz + 1) * F.nb[2] - 1) / d2;
            const int oy = gb.b[1], oz = gb.b[2];
            own_row = by == oy && bz == oz;
            const bool later = bz > oz || (bz == oz && by > oy);
            mine = own_row || (((by + bz + oy + oz) & 1) != 0) == later;
        }
        // segment k of [xa, xb]: wrapped below (k = 0), inside (1), wrapped above (2)
        const int a = k == 0 ? xa + d0 : (k == 1 ? max(xa, 0) : max(0, xa - d0));
        const int b = k == 0 ? min(d0 - 1, xb + d0) : (k == 1 ? min(xb, d0 - 1) : xb - d0);
        if (a <= b && (k != 0 || xa < 0) && (k != 2 || xb >= d0) && (mine || k != 1))
        {
            const uint32_t base =
                F.cell_base + static_cast<uint32_t>(d0 * ((uy - wy * d1) + d1 * (uz - wz * d2)));
            st = start[base + a];
            const uint32_t en = start[base + b + 1];
            wrap = k + 3 * (wy + 1) + 9 * (wz + 1);
            if (own_row && k == 1)
            {
                st = max(st, min(en, gd.after + 1));
                wrap |= RUN_OWN;
            }
            cnt = en - st;
        }
    }
    StencilRuns r;
    r.wrap = wrap;
    const uint32_t incl = warp_inclusive(cnt, lane);
    r.off = incl - cnt;
    r.first = st - r.off;
    r.total = __shfl_sync(GR_FULL, incl, 31);
    r.plain = !__any_sync(GR_FULL, cnt != 0 && (wrap & (RUN_OWN - 1)) != 13);
    return r;
}

} // namespace
} // namespace fg
