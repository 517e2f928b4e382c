// Fused ball query + RDF histogram over every frame of a batch: persistent warps
// take query groups (fg_groups.cuh) from a device counter, stream the group's
// stencil past them and add each counted pair to the block's shared histogram,
// flushed once per block with 64-bit atomics.
//
// Half stencil, for frames whose queries are their points (exclude_ii) and whose
// points all lie in the box: a pair of image 0 is tested once, from the end that
// stencil_runs picks, and counted twice - p_i - (p_j + 0) is exactly
// -(p_j - (p_i + 0)), so both bonds fall in one bin. A pair across the periodic boundary is met
// from both ends (r_ij = p_j - (p_i + v_k), r_ji = p_i - (p_j + v_-k)) and each end
// counted once. Other frames meet the whole stencil and count every bond once.
//
// Bound by instruction issue (75% issue active, ALU pipe 51%): about 18 warp
// instructions per candidate and group, of which 6 are the packed float arithmetic (two
// candidates an instruction, each operation rounded on its own) and 7 the bin's address,
// the range and slot tests and the shared add. 64 uneven frames (18.3 M points, density
// 0.85, r_max 4, 200 bins) 16.9 -> 11.0 ms and 4.2 M points in Gaussian blobs (r_max 5)
// 6.5 -> 4.0 ms against a block per cell with octant lists of candidates. Registers are
// held to 64 (32 warps an SM: 24 warps of more registers took 12.2, 40 of fewer 11.3 ms)
// and the code is kept short, each stage at one site: with the sweeps inlined at several
// sites the instruction cache missed on most issues and the 64 frames took 31 ms.
#include "fg_groups.cuh"
#include "fg_prof.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace fg {

namespace {

constexpr uint32_t HIST_WORDS_MAX = 4096; // shared histogram words of a block (two a bin and copy)

// Regular-axis bin of a counted pair (Histogram.h:327-351), every step rounded as
// the reference rounds it.
__device__ __noinline__ uint32_t exact_bin(const HistParams& h, float rsq)
{
    const uint32_t bin = static_cast<uint32_t>(__fmul_rn(__fsub_rn(__fsqrt_rn(rsq), h.h_min), h.h_inv));
    return bin < h.bins ? bin : h.bins - 1;
}

constexpr float AP_MAGIC = 12582912.0f; // 1.5 2^23: x + AP_MAGIC has round(x) in its low mantissa bits
constexpr uint32_t AP_MAGIC_BITS = 0x4b400000u;

__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

constexpr int HB_N = GR_BUF + 4; // room for the padding of the last four candidates

// Buffered candidates, a component per array so two neighbours load as one pair.
struct HistCands
{
    float x[HB_N], y[HB_N], z[HB_N];
    uint32_t s[HB_N]; // slot + 1
};

// A warp's buffers: candidates of image 0 for queries in the box, and others, with the
// negated image vector (groups with a query off the box: every candidate, with the
// image a query in the box would need, k + n_q, as three floats).
struct alignas(16) HistBuf
{
    HistCands zero, other;
    float vx[HB_N], vy[HB_N], vz[HB_N];
    uint32_t edges; // pairs of the current sweep near a bin edge
    uint32_t none;  // takes the increments of pairs that are not counted
    // the current group (kept here for the registers)
    GroupBox gb;
    GroupBounds gd;
    StencilRows rows;
};
static_assert(sizeof(HistBuf) % 16 == 0 && sizeof(HistCands) % 16 == 0 && HB_N % 4 == 0,
              "candidate arrays are read 16 bytes at a time");

// (No memory clobber: the histogram words are read after a barrier only, and loads of
// the candidate buffers may move past the increments.)
__device__ __forceinline__ void shared_increment(uint32_t address)
{
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(address));
}

// Where a warp's pairs go: shared histogram words (by shared address) [once, once +
// bins) counted once and the next bins words counted twice; once == 0: the global
// histogram (bins past the shared one's capacity).
struct HistSink
{
    uint32_t once;
    unsigned long long* global;

    __device__ __forceinline__ void add(const HistParams& h, uint32_t bin, bool two) const
    {
        if (once != 0)
            shared_increment(once + 4u * (bin + (two ? h.bins : 0u)));
        else
            atomicAdd(global + bin, two ? 2ull : 1ull);
    }
};

template<bool LOW> __device__ __forceinline__ bool counted(const HistParams& h, float rsq)
{
    return rsq < h.ap_b && (!LOW || rsq >= h.ap_a);
}

enum SweepMode
{
    SW_ZERO = 0,  // image 0: r = p_j - q
    SW_SHIFT = 1, // one image per candidate: r = p_j - (q + v)
    SW_PAIR = 2,  // the image is the pair's: k = (k + n_q) - n_q, any axis of |k| > 1 no pair
};

// The lane's query: position (w: the packed box image it lies in) and the slot test
// (candidates of slots up to own are not met; SW_PAIR: the one equal to own).
struct HistQuery
{
    float4 p;
    uint32_t own;

    __device__ __forceinline__ float image(int axis) const
    {
        return static_cast<float>(img_ax(__float_as_int(p.w), axis));
    }
};

// The rare part of sweep(): every counted pair (edge_only false, histograms past the
// shared one's capacity or bins too fine for the approximate root) or those near a bin
// edge, binned by the exact arithmetic. Kept out of line: the sweeps' own code has to
// stay in the instruction cache.
template<bool LOW, int MODE>
__device__ __noinline__ void sweep_exact(const HistParams& h, HistSink sink, const HistBuf& B, const DevBox& box,
                                         uint32_t n, HistQuery Q, bool two, bool edge_only)
{
    const HistCands& C = MODE == SW_ZERO ? B.zero : B.other;
    const float4 q = Q.p;
#pragma unroll 1
    for (uint32_t e = 0; e < n; ++e)
    {
        float qx = q.x, qy = q.y, qz = q.z;
        bool ok = C.s[e] > Q.own;
        if (MODE == SW_SHIFT) // v is stored negated
        {
            qx = __fsub_rn(qx, B.vx[e]);
            qy = __fsub_rn(qy, B.vy[e]);
            qz = __fsub_rn(qz, B.vz[e]);
        }
        if (MODE == SW_PAIR)
        {
            const float kx = B.vx[e] - Q.image(0), ky = B.vy[e] - Q.image(1), kz = B.vz[e] - Q.image(2);
            ok = fmaxf(fmaxf(fabsf(kx), fabsf(ky)), fabsf(kz)) <= 1.0f && C.s[e] != Q.own;
            const float* v = box.img[ok ? static_cast<int>(kx * 9.0f + ky * 3.0f + kz) + 13 : 13];
            qx = __fadd_rn(qx, v[0]);
            qy = __fadd_rn(qy, v[1]);
            qz = __fadd_rn(qz, v[2]);
        }
        const float rsq = dot3(__fsub_rn(C.x[e], qx), __fsub_rn(C.y[e], qy), __fsub_rn(C.z[e], qz));
        ok = ok && counted<LOW>(h, rsq);
        if (edge_only)
        {
            const float t = __fmaf_rn(sqrt_approx(rsq), h.h_inv, h.ap_c);
            ok = ok && fabsf(__fsub_rn(t, __fsub_rn(__fadd_rn(t, AP_MAGIC), AP_MAGIC))) > h.ap_edge;
        }
        if (ok)
            sink.add(h, exact_bin(h, rsq), two);
    }
}

// Every lane's query against the n buffered candidates of the mode. two: counted twice.
//
// Bin of a counted pair: t = (sqrt(r^2) - h_min) / width - 1/2 from the approximate
// root, the bin its nearest integer (adding 1.5 2^23 leaves it in the low mantissa
// bits). Within the stated margin of a bin edge (HistParams::ap_edge) the exact
// arithmetic decides: such pairs increment the warp's edge counter instead, and a
// sweep that met any (about one in twenty at 200 bins) goes over its candidates again
// for those alone. Pairs that are not counted increment a word of their own: a
// predicated shared add compiles to a branch with its convergence barrier, three
// instructions more than the two selects of the address.
template<bool LOW, int MODE>
__device__ __forceinline__ void sweep(const HistParams& h, const HistSink& sink, HistBuf& B, const DevBox& box,
                                      uint32_t n, const HistQuery& Q, bool two, int lane)
{
    __syncwarp();
    if (sink.once == 0 || h.ap == 0)
    {
        sweep_exact<LOW, MODE>(h, sink, B, box, n, Q, two, false);
        __syncwarp();
        return;
    }
    HistCands& C = MODE == SW_ZERO ? B.zero : B.other;
    if (lane < 3)
    {
        C.x[n + lane] = GR_FAR;
        C.s[n + lane] = 0;
        if (MODE != SW_ZERO)
            B.vx[n + lane] = 0.0f;
    }
    __syncwarp();
    const uint32_t base = sink.once + 4u * ((two ? h.bins : 0u) - AP_MAGIC_BITS);
    const uint32_t edges = static_cast<uint32_t>(__cvta_generic_to_shared(&B.edges));
    const float4 q = Q.p;
    const f32x2 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
    const f32x2 nz = h.neg_zero2;
    const f32x2 inv = pack2(h.h_inv, h.h_inv), off = pack2(h.ap_c, h.ap_c);
    const f32x2 magic = pack2(AP_MAGIC, AP_MAGIC), nmagic = pack2(-AP_MAGIC, -AP_MAGIC), neg1 = pack2(-1.0f, -1.0f);
    auto pair = [&](f32x2 cx, f32x2 cy, f32x2 cz, f32x2 vx, f32x2 vy, f32x2 vz, uint32_t s0, uint32_t s1) {
        // c - (q + v) = c + (-q - v): negation is exact at every step
        f32x2 ux = nqx, uy = nqy, uz = nqz;
        bool in0 = true, in1 = true;
        if (MODE == SW_SHIFT)
        {
            ux = add2(nqx, vx);
            uy = add2(nqy, vy);
            uz = add2(nqz, vz);
        }
        if (MODE == SW_PAIR)
        {
            // -v = (-k1) a1 + (-k2) a2 + (-k3) a3, each product exact (|k| <= 1)
            const float *a1 = box.img[22], *a2 = box.img[16], *a3 = box.img[14];
            const float qi = Q.image(0), qj = Q.image(1), qk = Q.image(2);
            const f32x2 kx = fma2(vx, neg1, pack2(qi, qi)), ky = fma2(vy, neg1, pack2(qj, qj)),
                        kz = fma2(vz, neg1, pack2(qk, qk));
            ux = add2(nqx, fma2(kz, pack2(a3[0], a3[0]), fma2(ky, pack2(a2[0], a2[0]), fma2(kx, pack2(a1[0], a1[0]), nz))));
            uy = add2(nqy, fma2(kz, pack2(a3[1], a3[1]), fma2(ky, pack2(a2[1], a2[1]), nz)));
            uz = add2(nqz, fma2(kz, pack2(a3[2], a3[2]), nz));
            float x0, x1, y0, y1, z0, z1;
            unpack2(kx, x0, x1);
            unpack2(ky, y0, y1);
            unpack2(kz, z0, z1);
            in0 = fmaxf(fmaxf(fabsf(x0), fabsf(y0)), fabsf(z0)) <= 1.0f;
            in1 = fmaxf(fmaxf(fabsf(x1), fabsf(y1)), fabsf(z1)) <= 1.0f;
        }
        const f32x2 dx = add2(cx, ux), dy = add2(cy, uy), dz = add2(cz, uz);
        const f32x2 rr = add2(add2(fma2(dx, dx, nz), fma2(dy, dy, nz)), fma2(dz, dz, nz));
        float r0, r1, m0, m1, f0, f1;
        unpack2(rr, r0, r1);
        const f32x2 t = fma2(pack2(sqrt_approx(r0), sqrt_approx(r1)), inv, off);
        const f32x2 m = add2(t, magic);
        const f32x2 f = fma2(add2(m, nmagic), neg1, t);
        unpack2(m, m0, m1);
        unpack2(f, f0, f1);
        auto put = [&](float r, float m, float f, uint32_t slot, bool in) {
            const uint32_t at = fabsf(f) > h.ap_edge ? edges : base + 4u * __float_as_uint(m);
            const bool met = MODE == SW_PAIR ? in && slot != Q.own : slot > Q.own;
            shared_increment(met && counted<LOW>(h, r) ? at : edges + 4u);
        };
        put(r0, m0, f0, s0, in0);
        put(r1, m1, f1, s1, in1);
    };
#pragma unroll 1
    for (uint32_t e = 0; e < n; e += 4)
    {
        const ulonglong2 cx = *reinterpret_cast<const ulonglong2*>(C.x + e);
        const ulonglong2 cy = *reinterpret_cast<const ulonglong2*>(C.y + e);
        const ulonglong2 cz = *reinterpret_cast<const ulonglong2*>(C.z + e);
        const uint4 cs = *reinterpret_cast<const uint4*>(C.s + e);
        ulonglong2 vx = make_ulonglong2(0, 0), vy = vx, vz = vx;
        if (MODE != SW_ZERO)
        {
            vx = *reinterpret_cast<const ulonglong2*>(B.vx + e);
            vy = *reinterpret_cast<const ulonglong2*>(B.vy + e);
            vz = *reinterpret_cast<const ulonglong2*>(B.vz + e);
        }
        pair(cx.x, cy.x, cz.x, vx.x, vy.x, vz.x, cs.x, cs.y);
        pair(cx.y, cy.y, cz.y, vx.y, vy.y, vz.y, cs.z, cs.w);
    }
    __syncwarp();
    if (*static_cast<volatile uint32_t*>(&B.edges) != 0)
    {
        sweep_exact<LOW, MODE>(h, sink, B, box, n, Q, two, true);
        __syncwarp();
        *static_cast<volatile uint32_t*>(&B.edges) = 0; // (every lane, the same value)
    }
    __syncwarp();
}

// The sweep for groups with a query off the box, out of line (rare).
template<bool LOW>
__device__ __noinline__ void sweep_pairs(const HistParams& h, HistSink sink, HistBuf& B, const DevBox& box, uint32_t n,
                                         HistQuery Q, int lane)
{
    sweep<LOW, SW_PAIR>(h, sink, B, box, n, Q, false, lane);
}

// Places a round of candidates near the boundary, or of a frame with points off the box:
// c (w: packed image) of a cell with the given wrap. Returns the buffers' new counts.
__device__ __forceinline__ uint2 place_images(HistBuf& B, const DevBox& box, float cull2, float4 c, int wrap,
                                              uint32_t cslot, bool keep, bool qout, uint2 counts, int lane)
{
    const unsigned lt = (1u << lane) - 1u;
    // image for a query in the box: k = n_j - wrap (AABBQuery.cc:93,125)
    const int pim = __float_as_int(c.w);
    const int kx = img_ax(pim, 0) - (wrap % 3 - 1);
    const int ky = img_ax(pim, 1) - ((wrap / 3) % 3 - 1);
    const int kz = img_ax(pim, 2) - (wrap / 9 - 1);
    const bool zero = !qout && kx == 0 && ky == 0 && kz == 0;
    float vx = static_cast<float>(kx), vy = static_cast<float>(ky), vz = static_cast<float>(kz);
    if (!qout)
    {
        keep = keep && kx >= -1 && kx <= 1 && ky >= -1 && ky <= 1 && kz >= -1 && kz <= 1;
        const float* iv = box.img[keep ? 13 - kx * 9 - ky * 3 - kz : 13]; // of -k: negated
        vx = iv[0];
        vy = iv[1];
        vz = iv[2];
        keep = keep && group_gap2(B.gd, c.x + vx, c.y + vy, c.z + vz) <= cull2;
    }
    const unsigned mz = __ballot_sync(GR_FULL, keep && zero);
    const unsigned mn = __ballot_sync(GR_FULL, keep && !zero);
    if (keep)
    {
        HistCands& C = zero ? B.zero : B.other;
        const uint32_t e = zero ? counts.x + __popc(mz & lt) : counts.y + __popc(mn & lt);
        C.x[e] = c.x;
        C.y[e] = c.y;
        C.z[e] = c.z;
        C.s[e] = cslot;
        if (!zero)
        {
            B.vx[e] = vx;
            B.vy[e] = vy;
            B.vz[e] = vz;
        }
    }
    return make_uint2(counts.x + __popc(mz), counts.y + __popc(mn));
}

template<int WARPS, bool LOW>
__global__ void __launch_bounds__(WARPS * 32, 32 / WARPS)
    k_frames_hist(BatchGrid g, BallParams p, HistParams h, const uint4* __restrict__ items,
                  const uint32_t* __restrict__ n_items, uint32_t parts, int copies, uint32_t* __restrict__ queue,
                  unsigned long long* __restrict__ hist)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HistBuf& B = reinterpret_cast<HistBuf*>(smem_raw)[threadIdx.x >> 5];
    uint32_t* const words = reinterpret_cast<uint32_t*>(smem_raw + sizeof(HistBuf) * WARPS);
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (uint32_t t = threadIdx.x; t < 2 * h.bins * copies; t += WARPS * 32)
        words[t] = 0;
    if (lane == 0)
        B.edges = 0;
    __syncthreads();
    HistSink sink;
    sink.once = copies > 0 ? static_cast<uint32_t>(__cvta_generic_to_shared(words + 2 * h.bins * (warp % copies))) : 0u;
    sink.global = hist;
    const uint32_t total = *n_items * parts;
    for (;;)
    {
        uint32_t id = 0;
        if (lane == 0)
            id = atomicAdd(queue, 1u);
        id = __shfl_sync(GR_FULL, id, 0);
        if (id >= total)
            break;
        uint32_t part = 0;
        if (parts > 1)
        {
            part = id % parts;
            id = id / parts;
        }
        const uint4 it = items[id];
        const FrameDesc& F = g.fd[it.x];
        const GroupBox gb = group_box(F, it.y);
        __syncwarp();
        const uint32_t slot = group_slot(F, gb, g.start, it.z, lane);
        const bool live = static_cast<uint32_t>(lane) < it.w;
        HistQuery Q;
        Q.p = make_float4(3e30f, 3e30f, 3e30f, 0.0f); // dead lanes: every r^2 is infinite
        if (live)
            Q.p = g.cpos[slot];
        // in_box: every point of the frame has image 0. qout: some query of the group has
        // not; its candidates are neither clipped nor culled, and the image is the pair's
        const bool in_box = g.frame_out[it.x] == 0;
        const bool half = in_box && p.exclude_ii;
        const bool qout = __any_sync(GR_FULL, __float_as_int(Q.p.w) != 0);
        const float far = __int_as_float(0x7f800000);
        GroupBounds gd;
        gd.lo[0] = redux_min(live ? Q.p.x : far);
        gd.lo[1] = redux_min(live ? Q.p.y : far);
        gd.lo[2] = redux_min(live ? Q.p.z : far);
        gd.hi[0] = redux_max(live ? Q.p.x : -far);
        gd.hi[1] = redux_max(live ? Q.p.y : -far);
        gd.hi[2] = redux_max(live ? Q.p.z : -far);
        gd.cull = F.cull;
        gd.cull2 = F.cull2;
        gd.clip = !qout && !F.b.tilted;
        gd.half = half;
        gd.after = __reduce_min_sync(GR_FULL, live ? slot : ~0u);
        const float cull2 = F.cull2;
        uint32_t nz = 0, nn = 0; // buffered candidates
        Q.own = half || (qout && p.exclude_ii) ? slot + 1 : 0u;
        // whole stencil, queries in the box: each meets itself once, at distance 0 (coordinates that
        // are not finite, which come with image 0, at none)
        if (p.exclude_ii && !half && !qout && part == 0 && counted<LOW>(h, 0.0f))
        {
            const float self = dot3(__fsub_rn(Q.p.x, Q.p.x), __fsub_rn(Q.p.y, Q.p.y), __fsub_rn(Q.p.z, Q.p.z));
            const unsigned met = __ballot_sync(GR_FULL, live && self == 0.0f);
            if (lane == 0)
                atomicAdd(hist + exact_bin(h, 0.0f), 0ull - __popc(met));
        }
        // one site each for the next chunk of the stencil, the next round of 32 candidates
        // and the two sweeps (a buffer is swept once it holds 32, and at the end); of
        // several parts each takes every parts-th round
        const StencilRows rows = stencil_rows(F, gb, gd);
        if (lane == 0)
        {
            B.gb = gb;
            B.gd = gd;
            B.rows = rows;
        }
        __syncwarp();
        const int per_chunk = rows_per_chunk(rows);
        int row0 = -per_chunk;
        StencilRuns R;
        R.total = 0;
        uint32_t base = 0, skip = part * 32;
        for (bool done = false; !done;)
        {
            if (base >= R.total)
            {
                row0 += per_chunk;
                done = row0 >= B.rows.n;
                if (!done)
                {
                    R = stencil_runs(F, B.gb, B.rows, g.start, row0, B.gd, lane);
                    base = skip;
                    // rounds of the chunk up to the next of this part past its end
                    const uint32_t rounds = (R.total + 31) / 32;
                    if (parts > 1)
                        skip = (skip / 32 + parts * 64 - rounds % parts) % parts * 32;
                    if (base >= R.total)
                        continue;
                }
            }
            if (!done)
            {
                const uint32_t t = base + static_cast<uint32_t>(lane);
                const int r = warp_run_of(R.off, t);
                const uint32_t cs = __shfl_sync(GR_FULL, R.first, r) + t;
                const int wr = __shfl_sync(GR_FULL, R.wrap, r);
                // candidates of other rows of boxes meet every query
                const uint32_t cslot = half && !(wr & RUN_OWN) ? ~0u : cs + 1;
                bool keep = t < R.total;
                base += 32 * parts;
                float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
                if (keep)
                    c = g.cpos[cs];
                if (in_box && R.plain)
                {
                    keep = keep && group_gap2(B.gd, c.x, c.y, c.z) <= cull2;
                    const unsigned m = __ballot_sync(GR_FULL, keep);
                    if (keep)
                    {
                        const uint32_t e = nz + __popc(m & lt);
                        B.zero.x[e] = c.x;
                        B.zero.y[e] = c.y;
                        B.zero.z[e] = c.z;
                        B.zero.s[e] = cslot;
                    }
                    nz += __popc(m);
                }
                else
                {
                    const uint2 now = place_images(B, F.b, cull2, c, wr & (RUN_OWN - 1), cslot, keep, qout,
                                                   make_uint2(nz, nn), lane);
                    nz = now.x;
                    nn = now.y;
                }
            }
            // image 0, every query in the box: q + 0 is q (up to the sign of a zero, which
            // r^2 does not see), so r = p_j - q
            if (nz >= 32 || (done && nz > 0))
            {
                sweep<LOW, SW_ZERO>(h, sink, B, F.b, nz, Q, half, lane);
                nz = 0;
            }
            if (nn >= 32 || (done && nn > 0))
            {
                if (!qout)
                    sweep<LOW, SW_SHIFT>(h, sink, B, F.b, nn, Q, false, lane);
                else
                    sweep_pairs<LOW>(h, sink, B, F.b, nn, Q, lane);
                nn = 0;
            }
        }
    }
    if (copies > 0)
    {
        __syncthreads();
        for (uint32_t bin = threadIdx.x; bin < h.bins; bin += WARPS * 32)
        {
            unsigned long long v = 0;
            for (int k = 0; k < copies; ++k)
                v += words[2 * k * h.bins + bin] + 2ull * words[(2 * k + 1) * h.bins + bin];
            if (v != 0)
                atomicAdd(&hist[bin], v);
        }
    }
}

template<int WARPS, bool LOW>
void hist_launch(const BatchGrid& g, const BallParams& p, const HistParams& h, const uint4* items,
                 const uint32_t* n_items, uint32_t expected, int copies, uint32_t* queue, unsigned long long* hist,
                 cudaStream_t s)
{
    static int sms = 0, resident = 0;
    const size_t most = sizeof(HistBuf) * WARPS + sizeof(uint32_t) * HIST_WORDS_MAX;
    if (sms == 0)
    {
        int dev = 0, per = 0, count = 0;
        cudaFuncSetAttribute(k_frames_hist<WARPS, LOW>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_frames_hist<WARPS, LOW>, WARPS * 32, most);
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        resident = std::max(1, per);
        sms = std::max(1, count);
    }
    const size_t smem = sizeof(HistBuf) * WARPS + sizeof(uint32_t) * 2 * h.bins * copies;
    // few groups: each is split over up to 12 warps by rounds of its candidates, until
    // every SM has 96 (10,000 points at density 1, r_max 4: 54 us unsplit by 3, 43 by 6,
    // 37 by 12; 100,000: 150 us unsplit, 122 by 3, 134 by 8)
    const uint32_t want = static_cast<uint32_t>(sms) * 96u;
    const uint32_t parts = std::min<uint32_t>(12u, std::max<uint32_t>(1u, want / std::max<uint32_t>(1u, expected)));
    const uint32_t blocks =
        std::min<uint32_t>(static_cast<uint32_t>(sms * resident),
                           std::max<uint32_t>(1u, (expected * parts + WARPS - 1) / WARPS));
    ProfScope prof_("k_frames_hist", s);
    k_frames_hist<WARPS, LOW><<<blocks, WARPS * 32, smem, s>>>(g, p, h, items, n_items, parts, copies, queue, hist);
}

// Small systems without tilt: every ordered pair, no grid. A warp holds 32 queries (a lane
// each) and meets a chunk of the points; of the images of a pair the nearest is the one that
// can be counted (2 r_max below every box length, with room for the rounding), and along
// each axis it is the smallest of |p - q|, |p - (q + L)| and |p - (q - L)|, each rounded as the
// AABB arithmetic rounds it. About 35 warp instructions for 32 pairs, which costs less than
// the latency of the grid, its groups and their tables up to SMALL_RDF_N points at every r_max: whole
// calls at density 1, r_max 0.4 to 6: 1000 points 81 to 84 us against 104 to 118, 3000 89 to 96 / 111
// to 143, 5000 106 to 121 / 118 to 147.
constexpr int SM_WARPS = 8;
constexpr int SM_CHUNK = 64; // at most

template<bool LOW>
__global__ void __launch_bounds__(SM_WARPS * 32)
    k_small_hist(DevBox b, const float* __restrict__ pts, uint32_t n, uint32_t chunk, int exclude_ii, HistParams h,
                 unsigned long long* __restrict__ hist)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4* const cand = reinterpret_cast<float4*>(smem_raw) + SM_CHUNK * (threadIdx.x >> 5);
    uint32_t* const counts = reinterpret_cast<uint32_t*>(smem_raw + sizeof(float4) * SM_CHUNK * SM_WARPS);
    const int lane = threadIdx.x & 31;
    for (uint32_t k = threadIdx.x; k < h.bins; k += SM_WARPS * 32)
        counts[k] = 0;
    __syncthreads();
    const uint32_t chunks = (n + chunk - 1) / chunk;
    const uint32_t units = (n + 31) / 32 * chunks;
    for (uint32_t u = blockIdx.x * SM_WARPS + (threadIdx.x >> 5); u < units; u += gridDim.x * SM_WARPS)
    {
        const uint32_t i = u / chunks * 32 + lane;
        const uint32_t j0 = u % chunks * chunk;
        const uint32_t nj = min(n - j0, chunk);
        __syncwarp();
        for (uint32_t e = lane; e < nj; e += 32)
        {
            const float* p = pts + 3 * static_cast<size_t>(j0 + e);
            cand[e] = make_float4(p[0], p[1], b.is2d ? 0.0f : p[2], 0.0f);
        }
        float q[3] = {3e30f, 3e30f, 3e30f}; // no query: every r^2 is infinite
        if (i < n)
        {
            const float* p = pts + 3 * static_cast<size_t>(i);
            q[0] = p[0];
            q[1] = p[1];
            q[2] = b.is2d ? 0.0f : p[2];
        }
        // the images +1 and -1 of each axis: codes 13 +- 9, 3, 1
        const float up[3] = {__fadd_rn(q[0], b.img[22][0]), __fadd_rn(q[1], b.img[16][1]), __fadd_rn(q[2], b.img[14][2])};
        const float dn[3] = {__fadd_rn(q[0], b.img[4][0]), __fadd_rn(q[1], b.img[10][1]), __fadd_rn(q[2], b.img[12][2])};
        const uint32_t own = exclude_ii ? i - j0 : 0xffffffffu;
        __syncwarp();
#pragma unroll 4
        for (uint32_t e = 0; e < nj; ++e)
        {
            const float4 p = cand[e];
            auto axis = [](float x, float q0, float q1, float q2) {
                return fminf(fminf(fabsf(__fsub_rn(x, q0)), fabsf(__fsub_rn(x, q1))), fabsf(__fsub_rn(x, q2)));
            };
            const float rsq = dot3(axis(p.x, q[0], up[0], dn[0]), axis(p.y, q[1], up[1], dn[1]),
                                   axis(p.z, q[2], up[2], dn[2]));
            if (counted<LOW>(h, rsq) && e != own)
            {
                const float t = __fmaf_rn(sqrt_approx(rsq), h.h_inv, h.ap_c);
                const float near = __fadd_rn(t, AP_MAGIC);
                uint32_t bin = __float_as_uint(near) - AP_MAGIC_BITS;
                if (h.ap == 0 || fabsf(__fsub_rn(t, __fsub_rn(near, AP_MAGIC))) > h.ap_edge)
                    bin = exact_bin(h, rsq);
                atomicAdd(&counts[bin], 1u);
            }
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < h.bins; k += SM_WARPS * 32)
    {
        if (counts[k] != 0)
            atomicAdd(hist + k, static_cast<unsigned long long>(counts[k]));
    }
}

} // namespace

bool nearest_image_fits(const float L[3], bool tilted, bool is2d, float r_max)
{
    return !tilted && r_max < 0.499f * std::min(std::min(L[0], L[1]), is2d ? L[1] : L[2]);
}

bool small_hist_fits(const DevBox& b, uint32_t n, float r_max, uint32_t bins)
{
    return n <= SMALL_RDF_N && bins <= HIST_WORDS_MAX && nearest_image_fits(b.L, b.tilted != 0, b.is2d != 0, r_max);
}

void launch_small_hist(const DevBox& b, const float* pts, uint32_t n, int exclude_ii, const HistParams& h,
                       unsigned long long* hist, cudaStream_t s)
{
    if (n == 0)
        return;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // chunks that give every SM a block, in eighths of the largest
    sms = std::max(sms, 1);
    const uint32_t tiles = (n + 31) / 32, warps = static_cast<uint32_t>(sms) * SM_WARPS;
    const uint32_t chunk = std::min<uint32_t>(SM_CHUNK, (static_cast<uint32_t>(static_cast<uint64_t>(n) * tiles / warps) / 8 + 1) * 8);
    const uint32_t units = tiles * ((n + chunk - 1) / chunk);
    const uint32_t blocks = std::min<uint32_t>(static_cast<uint32_t>(sms) * 4, (units + SM_WARPS - 1) / SM_WARPS);
    const size_t smem = sizeof(float4) * SM_CHUNK * SM_WARPS + sizeof(uint32_t) * h.bins;
    ProfScope prof_("k_small_hist", s);
    if (h.ap_a > 0.0f)
        k_small_hist<true><<<blocks, SM_WARPS * 32, smem, s>>>(b, pts, n, chunk, exclude_ii, h, hist);
    else
        k_small_hist<false><<<blocks, SM_WARPS * 32, smem, s>>>(b, pts, n, chunk, exclude_ii, h, hist);
}

void launch_frames_hist(const BatchHistConfig& cfg, const BatchGrid& g, const BallParams& p, const HistParams& h,
                        const uint4* items, const uint32_t* n_items, uint32_t expected, uint32_t* queue,
                        unsigned long long* hist, cudaStream_t s)
{
    if (expected == 0)
        return;
    int copies = cfg.copies;
    if (2 * h.bins * static_cast<uint64_t>(copies) > HIST_WORDS_MAX)
        copies = 2 * static_cast<uint64_t>(h.bins) <= HIST_WORDS_MAX ? 1 : 0;
    auto go = [&](auto launch) { launch(g, p, h, items, n_items, expected, copies, queue, hist, s); };
    if (cfg.warps == 4)
        go(h.ap_a > 0.0f ? hist_launch<4, true> : hist_launch<4, false>);
    else
        go(h.ap_a > 0.0f ? hist_launch<8, true> : hist_launch<8, false>);
}

// ---------------------------------------------------------------------------
// Bins from an approximate square root
//
// A pair is counted when r_min^2 <= r^2 < r_max^2 and h_min <= sqrt(r^2) < h_max
// (the root correctly rounded). Every step is monotone in r^2, and so in the bits
// of the non-negative float r^2: the counted pairs are an interval of bit patterns
// [ap_a, ap_b), found here by bisection with the same float operations.
//
// Its bin (Histogram.h:327-351) is trunc(T), T = RN(RN(RN(sqrt(r^2)) - h_min) h_inv),
// clipped to the last bin. With u = 2^-24, X = (sqrt(r^2) - h_min) h_inv and H =
// |h_min h_inv|, T is within u (3 X + H) of X. The kernel takes t = fma(s, h_inv,
// ap_c), s = sqrt.approx (relative error at most 2^-23 by the PTX manual) and ap_c =
// RN(RN(-h_min h_inv) - 1/2): t is within u (2 (X + H) + 2 H + X + 2) of X - 1/2. So
// |t + 1/2 - T| <= u (6 X + 5 H + 2) <= u (6 bins + 5 H + 3) =: e, and when t lies farther than e from every half
// integer, trunc(T) is the integer nearest t. Nearer, the exact arithmetic decides
// (t - round(t) is exact; a few u are added below).
// ---------------------------------------------------------------------------
namespace {

constexpr uint32_t INF_BITS = 0x7f800000u;

float bits_float(uint32_t u)
{
    float f;
    std::memcpy(&f, &u, sizeof(float));
    return f;
}

// smallest u in [lo, hi) with pred(u), else hi; pred is false then true
template<typename P> uint32_t first_true(uint32_t lo, uint32_t hi, P pred)
{
    while (lo < hi)
    {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (pred(mid))
            hi = mid;
        else
            lo = mid + 1;
    }
    return lo;
}

} // namespace

HistParams with_approx_bins(const HistParams& h, float r_min_sq, float r_max_sq)
{
    HistParams out = h;
    const double shift = std::abs(static_cast<double>(h.h_min) * h.h_inv);
    const double e = (6.0 * h.bins + 5.0 * shift + 8.0) * 0x1p-24;
    const uint32_t ua = first_true(0u, INF_BITS + 1, [&](uint32_t u) {
        const float r = bits_float(u);
        return r >= r_min_sq && std::sqrt(r) >= h.h_min;
    });
    const uint32_t ub = first_true(0u, INF_BITS + 1, [&](uint32_t u) {
        const float r = bits_float(u);
        return r >= r_max_sq || std::sqrt(r) >= h.h_max;
    });
    // margins past an eighth of a bin would send a quarter of the pairs to the exact
    // arithmetic; the sum t + 1.5 2^23 needs t below 2^22
    out.ap = e <= 0.125 ? 1 : 0;
    out.ap_a = ua < ub ? bits_float(ua) : 0.0f;
    out.ap_b = ua < ub ? bits_float(ub) : 0.0f;
    out.ap_c = fsub(-fmul(h.h_min, h.h_inv), 0.5f);
    out.ap_edge = static_cast<float>(0.5 - e);
    out.neg_zero2 = NEG_ZERO2;
    return out;
}

} // namespace fg
