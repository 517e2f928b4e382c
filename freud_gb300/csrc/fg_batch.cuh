// Launch interface of the batched (many frames, one launch) kernels.
//
// A batch holds F frames of uneven N: points concatenated frame after frame,
// each frame with its own periodic box. One cell grid spans every frame: frame
// f owns the cells [cell_base[f], cell_base[f + 1]) and the points
// [pt_base[f], pt_base[f + 1]); point indices are global (into the
// concatenation), so per-point outputs of every frame land in one array.
// Pair arithmetic is the AABB arithmetic of a (box, points) system
// (AABBQuery.cc:93,125): r = p_j - (q + image_k), k = n_j - n_q - wrap.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "fg_kernels.cuh"
#include "fg_steinhardt.cuh"

namespace fg {

struct FrameDesc
{
    DevBox b;
    int dim[3];
    int shell;          // stencil half-width in cells: cells are >= r_max / shell wide
    uint32_t cell_base; // first cell of the frame in the batch grid
    uint32_t ncell;
    uint32_t pt_base;   // first point of the frame
    uint32_t n;
    // query groups (fg_groups.cuh): boxes of cells per axis, the frame's first box in
    // the batch, and the cull radius: r_max plus a margin bounding the difference between
    // the image-shifted float distance and the exact one
    int nb[3];
    uint32_t box_base;
    float cull, cull2;
    float cell_width[3], cells_per[3]; // box lengths / dim and dim / box lengths
};

// Cell grid over every frame of a batch.
struct BatchGrid
{
    const FrameDesc* fd;       // [nframes]
    const uint32_t* cell_base; // [nframes + 1]
    uint32_t nframes;
    uint32_t ncell;            // all frames
    const uint32_t* start;     // [ncell + 1] exclusive offsets into the point slots
    const float4* cpos;        // cell-sorted positions, w = packed integer box image
    const uint32_t* cidx;      // global point index of each slot
    const uint32_t* cell_of;   // global cell of each point (by point index)
    const int* frame_out;      // [nframes]: nonzero when some point of the frame lies outside its box
    const uint32_t* box_base;  // [nframes + 1] first box of cells of each frame
    uint32_t nboxes;           // all frames
};

// Tunable launch shape of the batched histogram kernel.
struct BatchHistConfig
{
    int shell;  // 1: 27-cell stencil of r_max cells; 2: 125-cell stencil of r_max / 2 cells
    int warps;  // warps per block (4 or 8)
    int copies; // privatised shared histograms per block (1, 2 or one per warp)
};

// Counting sort of every frame's points into the batch grid. cell_count must be
// zeroed ([ncell + 1]); pos4 receives (x, y, z, image) per point.
// frame_out ([nframes], zeroed) is set for each frame with a point outside its box.
void launch_frames_assign(const FrameDesc* fd, const uint32_t* pt_base, uint32_t nframes, const float* pts,
                          uint32_t n, uint32_t* cell_of, uint32_t* rank, float4* pos4, uint32_t* cell_count,
                          int* frame_out, cudaStream_t s);
void launch_frames_scatter(uint32_t n, const uint32_t* cell_of, const uint32_t* rank, const float4* pos4,
                           const uint32_t* start, float4* cpos, uint32_t* cidx, cudaStream_t s);

// Boxes of cells for a frame's query groups: nb boxes per axis over dim cells, sized
// for about one warp of points each. Returns how many groups uniform points make.
double group_boxes(const int dim[3], uint32_t n, int shell, int nb[3]);
double nl_boxes(const int dim[3], uint32_t nq, uint32_t np, double reach, int nb[3], double* met);
// Lists the query groups of the first nboxes boxes of the batch: items[i] = (frame,
// box of the frame, first point of the box's, points of the group), *n_items of them
// (zeroed before the launch; at most nboxes + n / 32 + 1). Boxes without points have
// none; a box's points are split evenly.
void launch_frames_groups(const BatchGrid& g, uint32_t nboxes, uint4* items, uint32_t* n_items, cudaStream_t s);

// The grid of one system of up to SMALL_N points and SMALL_CELLS cells by one block
// (fg_small_grid.cu), with its query groups where items is set. A system's own grid has at
// most 2 n + 64 cells, so its points decide; query points of their own are put into the cells of the
// points' grid, which may be any number. Both limits together fit the block's shared memory
// (131 KB) and 16 bits a cell. Up to there the block is the faster one, whole calls
// against the general build: RDF of 1000 points 99 / 112 us, 6000 108 / 114, 10000 116 / 118;
// Steinhardt 129 / 146, 136 / 148, 150 / 163; NeighborList 143 / 156, 184 / 186, 212 / 201.
constexpr uint32_t SMALL_N = 8192;
constexpr uint32_t SMALL_CELLS = 2 * SMALL_N + 64;
inline bool small_grid_fits(uint32_t n, uint64_t ncell)
{
    return n <= SMALL_N && ncell <= SMALL_CELLS;
}
struct SmallGrid
{
    FrameDesc F;         // box, dim, ncell; boxes of the query groups; cell_base 0
    const float* pts;
    uint32_t n;
    int sorted;          // each cell's points in index order
    uint32_t* start;     // [ncell + 1]
    float4* cpos;
    uint32_t* cidx;
    int* out;            // set to whether some point lies outside its box (or null)
    uint4* items;        // query groups (or null)
    uint32_t nboxes;
    uint32_t* words;     // words[0] = groups, the other n_words - 1 zeroed
    uint32_t n_words;
};
void launch_small_grid(const SmallGrid& a, cudaStream_t s);

// Fused ball query + RDF histogram over the listed query groups (fg_frames_hist.cu).
// expected: about how many groups there are (sizes the launch). *queue zeroed before
// the launch. hist is uint64[h.bins].
// h with the counted range of r^2 and the constants of the approximate-root binning
// filled in (the pair test r_min_sq <= r^2 < r_max_sq folded in).
HistParams with_approx_bins(const HistParams& h, float r_min_sq, float r_max_sq);
void launch_frames_hist(const BatchHistConfig& cfg, const BatchGrid& g, const BallParams& p, const HistParams& h,
                        const uint4* items, const uint32_t* n_items, uint32_t expected, uint32_t* queue,
                        unsigned long long* hist, cudaStream_t s);

// The histogram of one system of up to SMALL_RDF_N points without a grid: every pair
// (h from with_approx_bins).
constexpr uint32_t SMALL_RDF_N = 5120;
// Whether the nearest image of a pair is the one within r_max: no tilt, and r_max below half
// of every length with room for the rounding.
bool nearest_image_fits(const float L[3], bool tilted, bool is2d, float r_max);
bool small_hist_fits(const DevBox& b, uint32_t n, float r_max, uint32_t bins);
void launch_small_hist(const DevBox& b, const float* pts, uint32_t n, int exclude_ii, const HistParams& h,
                       unsigned long long* hist, cudaStream_t s);

// Ball query over every frame (grid of r_max cells, shell 1), warp per cell.
// Count pass: counts[i] = bonds of point i. Fill pass: bonds of point i at
// offsets[i] in candidate order: the neighbour index j and one float4 holding the
// Steinhardt bond vector box.wrap(p_j - p_i) (Steinhardt.cc:155) and the distance.
// *most (zeroed) = points of the fullest cell.
void launch_fullest_cell(const BatchGrid& g, uint32_t* most, cudaStream_t s);
// heavy: room for ball_heavy_items(n) groups of cells of many points, and their number.
struct BallHeavy
{
    uint2* items;
    uint32_t* n;
};
size_t ball_heavy_items(uint32_t n);
void launch_frames_ball_count(const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                              uint32_t* counts, cudaStream_t s);
void launch_frames_ball_fill(const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                             const uint64_t* offsets, uint32_t* bond_j, float4* bond_vd, cudaStream_t s);
// One pass without the counts: warps take chunks of the bond arrays (capacity
// cap) from *alloc (zeroed before the launch); seg[i] / counts[i] = the first bond
// of point i and its bond count, its bonds in candidate order. *alloc > cap after
// the launch: the arrays were too small and nothing past cap was written.
uint64_t frames_ball_onepass_slack(uint32_t ncell, uint32_t n); // bond slots the chunk tails may leave unused
void launch_frames_ball_onepass(const BatchGrid& g, const BallParams& p, uint32_t n, const BallHeavy& heavy,
                                uint32_t* counts, uint32_t* seg, uint32_t* bond_j, float4* bond_vd,
                                unsigned long long* alloc, uint64_t cap, cudaStream_t s);

// q_lm of every point from the ball query, for single l up to FRAME_QLM_MAX_L
// (fg_frames_qlm.cu), with the neighbour averaging when list is set.
constexpr int FRAME_QLM_MAX_L = 12;
struct FrameQlm
{
    const uint4* items;       // query groups (launch_frames_groups)
    const uint32_t* n_items;
    uint32_t* queue;          // work counters, one per l, zeroed
    uint32_t expected;        // about how many groups
    const StLs* ls;
    float2* qlm;              // per l (n, 2l + 1) by point
    float* ql;                // (n, nl)
    float* rows;              // compact rows of the current l by slot: n * frame_row_floats(l)
    bool list;                // averaging
    float* rows_ave;          // its compact rows
    float* ql_ave;
    uint32_t* head;           // bond lists: first segment of each group,
    uint32_t* segs;           // segments (cap words),
    unsigned long long* alloc; // words taken (zeroed); more than cap: run again with room
    uint64_t cap;
};
int frame_row_floats(int l);
// Words of the bond lists for about groups query groups of bonds_per_point bonds a point.
uint64_t frame_segment_words(double groups, double bonds_per_point, uint32_t expected);
// The k-th l of w.ls (k = 0 first: it writes the bond lists).
void launch_frames_qlm(const BatchGrid& g, const BallParams& p, const FrameQlm& w, int k, cudaStream_t s);
// The same for one system of up to SMALL_ST_N points without a grid (nearest_image_fits), with
// the averaging where nb is set: every l of ls in turn.
constexpr uint32_t SMALL_ST_N = 3072;
constexpr uint32_t SMALL_ST_BONDS = 64; // neighbours of a particle listed for the averaging
struct SmallQlm
{
    DevBox b;
    const float* pts;
    uint32_t n;
    BallParams p;
    const StLs* ls;
    float2* qlm;
    float* ql;
    float* rows;              // n * frame_row_floats of the largest l
    uint32_t* nb;             // averaging: n * SMALL_ST_BONDS (or null)
    uint32_t* nb_count;       // n
    float* rows_ave;
    float* ql_ave;
    int* over;                // zeroed: set if some particle has more neighbours
    double* sys;              // system sums over n, the columns of every l
};
void launch_small_qlm(const SmallQlm& w, cudaStream_t s);
// System sums of one l from compact rows: the l's columns of partial (launch_frames_sys).
void launch_rows_sys(const uint32_t* pt_base, uint32_t nframes, uint32_t max_rows, int l, int stride, int col0,
                     const float* rows, double* partial, cudaStream_t s);
// The partial sums of every column reduced and divided by n_f.
void launch_frames_sys_final(const uint32_t* pt_base, uint32_t nframes, uint32_t max_rows, int stride,
                             const double* partial, double* sys, cudaStream_t s);

// k nearest neighbours of one system in query groups (fg_knn_groups.cu): 1 <= k <= 32, AABB
// arithmetic, no r_max or r_min, at least k points a query, shell 2, fewer than 2^27 points.
struct KnnGroups
{
    const uint4* items;       // room for the query groups
    const uint32_t* n_items;  // zeroed
    uint32_t* queue;          // zeroed
    uint32_t* fail;           // queries (by sorted position) the groups did not settle
    uint32_t* n_fail;         // zeroed
    const float* pts;         // the points by index (n x 3)
    uint32_t k;
    int exclude_ii, by_distance, flat;
    float target;             // points expected within the radius (knn_target)
    float covered;            // largest radius the shell covers, below half the smallest plane distance
    float cell_volume, margin;
    unsigned long long neg_zero2;
};
double knn_target(uint32_t k);
// Writes the rows of every query but the n_fail2 left in fail2 (sorted positions), and the
// list's segments.
void launch_knn_groups(const FrameDesc& F, const DevGrid& g, uint32_t nboxes, const uint32_t* qstart, const float4* qpos,
                       const uint32_t* qidx, const KnnGroups& params, uint32_t expected, float cell_width,
                       float half_min_plane, uint32_t nq, uint2* ij, float* dist, float* vec, uint32_t* seg, uint32_t* cnt,
                       uint32_t* fail2, uint32_t* n_fail2, cudaStream_t s);
void launch_knn_rows(const uint32_t* list, uint32_t nlist, const uint32_t* qidx, uint32_t k, int by_distance,
                     const uint32_t* counts, const uint32_t* tj, const float* td, const float* tv, uint2* ij, float* dist,
                     float* vec, uint32_t* n_short, cudaStream_t s);

// NeighborList of one system in query groups (fg_nl_groups.cu).
struct NlGroups
{
    const uint4* items;        // query groups
    const uint32_t* ids;       // those to take (null: all)
    const uint32_t* n_ids;     // how many
    uint32_t* queue;           // zeroed
    uint32_t* big;             // groups of more candidates than fit (null: their queries go to over)
    uint32_t* n_big;           // zeroed
    uint32_t* over;            // queries (by sorted position) left to the kernels a query at a time
    uint32_t* n_over;          // zeroed
    uint32_t* pool;            // segments: sorted candidates and acceptance bits
    unsigned long long* used;  // zeroed; units of 64 words taken; more than cap: run again with room
    unsigned long long cap;
    uint32_t* head;            // per group: its segment
    uint32_t* total;           // per group: its candidates
    uint32_t* counts;          // bonds per query
    float r_max, delta;        // delta: bound on the prefilter's difference from the exact distance
    float r_max_sq, r_min_sq;
    float half_min_plane;
    int exclude_ii;
    unsigned long long neg_zero2;
};
void launch_nl_items(const FrameDesc& F, uint32_t nboxes, const uint32_t* qstart, uint4* items, uint32_t* n_items,
                     cudaStream_t s);
// room: candidates of a group that fit (256, 512, 768 or 1024).
void launch_nl_groups(int room, bool wrap, bool wide_keys, const FrameDesc& F, const DevGrid& g, const uint32_t* qstart,
                      const float4* qpos, const uint32_t* qidx, const NlGroups& params, uint32_t expected, cudaStream_t s);
void launch_nl_groups_write(int room, bool wrap, const FrameDesc& F, const DevGrid& g, const uint32_t* qstart,
                            const float4* qpos, const uint32_t* qidx, const NlGroups& w, uint32_t expected,
                            const uint64_t* offsets, uint2* ij, float* dist, float* vec, cudaStream_t s);

// Per-frame FP64 system sums of the per-l (n, 2l + 1) qlm layout: sys[f][col]
// (complex, col running over every l's m) = (FP64 sum over the frame's rows) /
// n_f: float-float (exact TwoSum) running sums over runs of at most FRAME_SYS_ROWS
// rows, FP64 from there on (fixed shuffle trees, then a fixed tree over the runs),
// so results do not depend on scheduling. max_rows is the
// largest frame; partial holds nframes * frames_sys_splits(max_rows) * stride * 2
// doubles.
constexpr uint32_t FRAME_SYS_ROWS = 512;
int frames_sys_splits(uint32_t max_rows);
void launch_frames_sys(const uint32_t* pt_base, uint32_t nframes, uint32_t max_rows, const StLs& ls, int stride,
                       const float2* src, double* partial, double* sys, cudaStream_t s);

} // namespace fg
