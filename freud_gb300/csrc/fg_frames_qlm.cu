// Steinhardt q_lm of every frame of a batch straight from the ball query, for one l up
// to 12 at a time (float32): persistent warps take query groups (fg_groups.cuh); each
// lane keeps its own particle, finds the particle's bonds among the group's candidates
// and adds their harmonics in registers, so no bond list, no bond vectors and no
// cross-lane sums are needed. The neighbour averaging reads the neighbours' rows
// through bond lists laid out per group (below).
//
// Bound by instruction issue (66% issue active, 330 warp instructions a point: about a
// third the tests of the group's candidates, a third the harmonics, two bonds an
// instruction), 20 warps an SM (16 warps of more registers 7.6 ms, 24 of fewer 7.5 ms).
// 64 uneven frames, 18.3 M points, r_max 1.5, l = 6: q_lm 7.1 ms against 16.3 ms for a
// ball query that wrote 20 bytes a bond (a warp per cell, whose set-up few queries
// shared) and a kernel that read them back; averaging 4.5 -> 2.8 ms on half rows (m >= 0)
// in cell order. 4.2 M points in Gaussian blobs, r_max 1.2: 8.9 -> 2.7 ms.
//
// Bond vector box.wrap(p_j - p_i) and distance of the ball query (Steinhardt.cc:155-172);
// Y_l^m as in fg_steinhardt.cu (normalised Legendre recurrence in l for each m >= 0, the
// negative orders from Y_l^{-m} = (-1)^m conj(Y_l^m)).
#include "fg_groups.cuh"
#include "fg_prof.cuh"

#include <algorithm>
#include <cmath>
#include <utility>

namespace fg {

namespace {

constexpr int QW = 4;           // warps per block
constexpr int QB_CAP = 224;     // buffered candidates per warp
constexpr int QB_N = QB_CAP + 4;
constexpr int Q_ROWS = 64;      // listed bonds per lane before they are summed

// Compact row of one particle: re, im of m = 0 .. l, padded to 16 bytes.
__host__ __device__ constexpr int row_floats(int l)
{
    return (2 * (l + 1) + 3) / 4 * 4;
}

// ---- coefficients, in double at compile time -----------------------------------------
constexpr double c_sqrt(double x)
{
    double r = x > 1.0 ? x : 1.0;
    for (int k = 0; k < 60; ++k)
        r = 0.5 * (r + x / r);
    return r;
}

// Associated Legendre functions without their leading factors, T_l = (l - m)! P_l^m /
// P_m^m: T_l = (2l - 1) x T_{l-1} - (l + m - 1) (l - m - 1) T_{l-2}, T_m = 1, whose
// coefficients are whole numbers, exact in float32. Rounded ones (of a normalised
// recurrence) put 2.7e-8 of Y_00 into every Y_60, a bias that adds up over all bonds where
// q_lm itself averages out: the system order of 10^5 disordered particles loses a digit.
constexpr double c_step(int l, int m)
{
    return (l + m - 1.0) * (l - m - 1.0);
}

// Y_lm = front T_l (sin(theta) e^{i phi})^m:
// (-1)^m (2m - 1)!! sqrt((2l + 1) / (4 pi) (l - m)! / (l + m)!) / (l - m)!
constexpr double c_front(int l, int m)
{
    double f2 = (2.0 * l + 1.0) / (4.0 * 3.14159265358979323846);
    for (int t = 1; t <= m; ++t)
        f2 *= (2.0 * t - 1.0) * (2.0 * t - 1.0);
    for (int t = 1; t <= l - m; ++t)
        f2 /= t;
    for (int t = 1; t <= l + m; ++t)
        f2 /= t;
    // (the square root at a size near 1)
    double scale = 1.0;
    while (f2 < 1.0)
    {
        f2 *= 4.0;
        scale *= 0.5;
    }
    return c_sqrt(f2) * scale * ((m & 1) ? -1.0 : 1.0);
}

template<int L> struct Coef
{
    float step[L + 1][L + 1] = {}; // [m][l]
    float front[L + 1] = {};
    constexpr Coef()
    {
        for (int m = 0; m <= L; ++m)
        {
            for (int l = m + 2; l <= L; ++l)
                step[m][l] = static_cast<float>(c_step(l, m));
            front[m] = static_cast<float>(c_front(L, m));
        }
    }
};

struct alignas(16) QBuf
{
    float x[QB_N], y[QB_N], z[QB_N];
    float vx[QB_N], vy[QB_N], vz[QB_N]; // negated image vector; with a query off the box k + n_q
    uint32_t s[QB_N];                   // slot + 1
    unsigned char list[Q_ROWS][32];        // the lanes' accepted candidates
    GroupBox gb;
    GroupBounds gd;
    StencilRows rows;
};

// One axis of box.wrap of two bond vectors p_j - p_i in a box without tilt, in the same
// roundings as box_wrap: the points lie in the box, so the fractional coordinates lie in
// (-1, 2) and each fmod of Box::wrap is a compare (NEAR: pairs of image 0, in [0, 1]).
template<bool NEAR> __device__ __forceinline__ f32x2 wrap_axis2(const DevBox& b, int a, f32x2 v, f32x2 nz)
{
    const f32x2 d = add2(v, pack2(-b.lo[a], -b.lo[a]));
    const f32x2 y = pack2(b.rcp[a], b.rcp[a]), nl = pack2(-b.L[a], -b.L[a]);
    const f32x2 q0 = fma2(d, y, nz);
    const f32x2 q1 = fma2(fma2(q0, nl, d), y, q0);
    f32x2 f = fma2(fma2(q1, nl, d), y, q1);
    float x0, x1;
    if (!NEAR)
    {
        unpack2(f, x0, x1);
        f = add2(f, pack2(x0 >= 1.0f ? -1.0f : 0.0f, x1 >= 1.0f ? -1.0f : 0.0f));
    }
    const f32x2 g = add2(f, pack2(1.0f, 1.0f));
    unpack2(g, x0, x1);
    const f32x2 m = NEAR ? add2(g, pack2(x0 >= 2.0f ? -2.0f : -1.0f, x1 >= 2.0f ? -2.0f : -1.0f))
                         : add2(g, pack2(x0 >= 2.0f ? -2.0f : (x0 >= 1.0f ? -1.0f : 0.0f),
                                         x1 >= 2.0f ? -2.0f : (x1 >= 1.0f ? -1.0f : 0.0f)));
    return add2(fma2(m, pack2(b.L[a], b.L[a]), nz), pack2(b.lo[a], b.lo[a]));
}

// sum += the harmonics of two bonds: vectors w, squared distances r0, r1; on1: the
// second one counts. acc[2 m], acc[2 m + 1]: re, im of order m, the two bonds in halves.
template<int L>
__device__ __forceinline__ void add_harmonics(f32x2* acc, f32x2 wx, f32x2 wy, f32x2 wz, float r0, float r1, bool on1)
{
    constexpr Coef<L> C;
    const f32x2 one = pack2(1.0f, 1.0f), zero = 0ull;
    if (L == 0)
    {
        acc[0] = fma2(pack2(C.front[0], C.front[0]), pack2(1.0f, on1 ? 1.0f : 0.0f), acc[0]);
        return;
    }
    // d = RN(sqrt(r^2)), the distance that the angles are taken from (Steinhardt.cc:163-172;
    // from r^2 itself sin(theta) near the poles is off by d's rounding, 4e-5 of Y_61), and
    // cos(theta) = RN(z / d), each by a remainder from the approximate root; sin^2(theta) = 1
    // - cos^2 with the quotient's remainder, accurate at every angle. theta = 0 when d = 0
    // or |z| >= d.
    const f32x2 neg = pack2(-1.0f, -1.0f), half = pack2(0.5f, 0.5f);
    const f32x2 y0 = pack2(r0 > 0.0f ? rsqrtf(r0) : 0.0f, r1 > 0.0f ? rsqrtf(r1) : 0.0f);
    const f32x2 rr = pack2(r0, r1);
    const f32x2 d0 = fma2(rr, y0, zero);
    const f32x2 d = fma2(fma2(fma2(d0, neg, zero), d0, rr), fma2(y0, half, zero), d0);
    const f32x2 nd = fma2(d, neg, zero);
    const f32x2 y = fma2(fma2(nd, y0, one), y0, y0);
    const f32x2 q0 = fma2(wz, y, zero);
    const f32x2 cq = fma2(fma2(nd, q0, wz), y, q0);
    const f32x2 lo = fma2(fma2(nd, cq, wz), y, zero);
    const f32x2 ncq = fma2(cq, neg, zero);
    const f32x2 s2 = fma2(add2(ncq, ncq), lo, fma2(ncq, cq, one)); // sin^2
    float s20, s21, c0, c1, z0, z1, p0, p1;
    unpack2(s2, s20, s21);
    unpack2(cq, c0, c1);
    unpack2(wz, z0, z1);
    const bool up0 = s20 > 0.0f && r0 > 0.0f, up1 = s21 > 0.0f && r1 > 0.0f;
    c0 = up0 ? c0 : (z0 < 0.0f ? -1.0f : 1.0f);
    c1 = up1 ? c1 : (z1 < 0.0f ? -1.0f : 1.0f);
    const f32x2 ct = pack2(c0, c1);
    // sin(theta) e^{i phi} = (x, y) sin(theta) / sqrt(x^2 + y^2): from the approximate root, then
    // the rounded vector's norm corrected to sin(theta) (its powers would carry m times the
    // error; rms of Y_66 5e-8, 1.1e-7 without)
    const f32x2 rho2 = fma2(wx, wx, fma2(wy, wy, zero));
    unpack2(fma2(s2, rho2, zero), p0, p1);
    const bool far0 = p0 > 1e-30f, far1 = p1 > 1e-30f;
    const f32x2 f = fma2(s2, pack2(up0 && far0 ? rsqrtf(p0) : 0.0f, up1 && far1 ? rsqrtf(p1) : 0.0f), zero);
    const f32x2 hx = fma2(wx, f, zero), hy = fma2(wy, f, zero);
    const f32x2 nhx = fma2(hx, neg, zero), nhy = fma2(hy, neg, zero);
    const f32x2 off = fma2(nhy, hy, fma2(nhx, hx, s2));
    const f32x2 k = fma2(off, pack2(up0 && far0 ? __fdividef(0.5f, s20) : 0.0f, up1 && far1 ? __fdividef(0.5f, s21) : 0.0f),
                         zero);
    f32x2 ex = fma2(hx, k, hx), ey = fma2(hy, k, hy);
    if ((up0 && !far0) || (up1 && !far1))
    {
        // on the axis or next to it: x, y scaled; e^{i phi} = 1 when both are 0
        auto near = [](float s, float u, float v, float& e, float& g) {
            u *= 1.1529215e18f; // 2^60
            v *= 1.1529215e18f;
            const float w = sqrtf(u * u + v * v), t = sqrtf(s);
            e = w > 0.0f ? u / w * t : t;
            g = w > 0.0f ? v / w * t : 0.0f;
        };
        float x0, x1, v0, v1, e0, e1, g0, g1;
        unpack2(wx, x0, x1);
        unpack2(wy, v0, v1);
        unpack2(ex, e0, e1);
        unpack2(ey, g0, g1);
        if (up0 && !far0)
            near(s20, x0, v0, e0, g0);
        if (up1 && !far1)
            near(s21, x1, v1, e1, g1);
        ex = pack2(e0, e1);
        ey = pack2(g0, g1);
    }
    const f32x2 on = pack2(1.0f, on1 ? 1.0f : 0.0f);
    f32x2 x[L + 1]; // (2 l - 1) cos(theta)
#pragma unroll
    for (int l = 1; l <= L; ++l)
        x[l] = l == 1 ? ct : fma2(ct, pack2(2.0f * l - 1.0f, 2.0f * l - 1.0f), zero);
    f32x2 zr = one, zi = zero; // (sin(theta) e^{i phi})^m
    const f32x2 ney = fma2(ey, pack2(-1.0f, -1.0f), zero);
#pragma unroll
    for (int m = 0; m <= L; ++m)
    {
        if (m == 1)
        {
            zr = ex;
            zi = ey;
        }
        else if (m > 1)
        {
            const f32x2 nr = fma2(zi, ney, fma2(zr, ex, zero));
            zi = fma2(zr, ey, fma2(zi, ex, zero));
            zr = nr;
        }
        f32x2 prev = one, cur = m < L ? x[m < L ? m + 1 : L] : one;
#pragma unroll
        for (int l = m + 2; l <= L; ++l)
        {
            const float c = -C.step[m][l];
            const f32x2 r = fma2(x[l], cur, l == m + 2 ? pack2(c, c) : fma2(prev, pack2(c, c), zero));
            prev = cur;
            cur = r;
        }
        const f32x2 q = fma2(fma2(cur, pack2(C.front[m], C.front[m]), zero), on, zero);
        acc[2 * m] = fma2(q, zr, acc[2 * m]);
        if (m > 0)
            acc[2 * m + 1] = fma2(q, zi, acc[2 * m + 1]);
    }
}

// Bond lists for the averaging, LIST: a segment per sweep of a group - 32 bond counts,
// 32 slots, the group's next segment (0: none) and padding to 96 words, then rows of 32
// neighbour slots (row k, lane t: bond k of the lane's particle). head[item]: the
// group's first segment, in words + 1 (0: none).
constexpr uint32_t SEG_HEAD = 96;
constexpr uint32_t SEG_CHUNK = 16384; // words a warp takes at a time

template<int L, bool LIST>
__global__ void __launch_bounds__(QW * 32, 5)
    k_frames_qlm(BatchGrid g, BallParams p, unsigned long long neg_zero2, const uint4* __restrict__ items,
                 const uint32_t* __restrict__ n_items, uint32_t* __restrict__ queue, float norm, int nl, int k_out,
                 float2* __restrict__ qlm, float* __restrict__ ql, float* __restrict__ rows_out,
                 uint32_t* __restrict__ head, uint32_t* __restrict__ segs, unsigned long long* __restrict__ alloc,
                 unsigned long long cap)
{
    constexpr int RS = row_floats(L);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    QBuf& B = reinterpret_cast<QBuf*>(smem_raw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t total = *n_items;
    unsigned long long cur = 0, cend = 0; // the warp's chunk of the segments
    for (;;)
    {
        uint32_t id = 0;
        if (lane == 0)
            id = atomicAdd(queue, 1u);
        id = __shfl_sync(GR_FULL, id, 0);
        if (id >= total)
            break;
        const uint4 it = items[id];
        const FrameDesc& F = g.fd[it.x];
        const DevBox& box = F.b;
        const bool in_box = g.frame_out[it.x] == 0; // every point of the frame
        bool plain, qout;
        uint32_t slot;
        float4 q = make_float4(3e30f, 3e30f, 3e30f, 0.0f); // dead lanes: every r^2 is infinite
        {
            const GroupBox gb = group_box(F, it.y);
            slot = group_slot(F, gb, g.start, it.z, lane);
            const bool live = static_cast<uint32_t>(lane) < it.w;
            if (live)
                q = g.cpos[slot];
            qout = __any_sync(GR_FULL, __float_as_int(q.w) != 0);
            const float far = __int_as_float(0x7f800000);
            GroupBounds gd;
            gd.lo[0] = redux_min(live ? q.x : far);
            gd.lo[1] = redux_min(live ? q.y : far);
            gd.lo[2] = redux_min(live ? q.z : far);
            gd.hi[0] = redux_max(live ? q.x : -far);
            gd.hi[1] = redux_max(live ? q.y : -far);
            gd.hi[2] = redux_max(live ? q.z : -far);
            gd.cull = F.cull;
        gd.cull2 = F.cull2;
        gd.clip = !qout && !box.tilted;
            gd.half = false;
            gd.after = 0;
            const StencilRows rows = stencil_rows(F, gb, gd);
            __syncwarp();
            if (lane == 0)
            {
                B.gb = gb;
                B.gd = gd;
                B.rows = rows;
            }
            __syncwarp();
            // every candidate of image 0 (with points in the box): none across the boundary
            const int s = F.shell;
            plain = in_box && rows.segs == 1 && gb.lo[1] >= s && gb.hi[1] + s <= F.dim[1] &&
                (box.is2d || (gb.lo[2] >= s && gb.hi[2] + s <= F.dim[2]));
        }
        const uint32_t own = p.exclude_ii ? slot + 1 : 0u;
        const float cull2 = F.cull2;
        const f32x2 nz = neg_zero2;
        const f32x2 nqx = pack2(-q.x, -q.x), nqy = pack2(-q.y, -q.y), nqz = pack2(-q.z, -q.z);
        f32x2 acc[2 * (L + 1)];
#pragma unroll
        for (int v = 0; v < 2 * (L + 1); ++v)
            acc[v] = 0ull;
        uint32_t bonds = 0, n = 0; // bonds summed, candidates buffered
        uint32_t prev_next = 0;    // LIST: word + 1 of the last segment's link
        if (LIST && lane == 0)
            head[id] = 0;

        const int per_chunk = rows_per_chunk(B.rows);
        int row0 = -per_chunk;
        StencilRuns R;
        R.total = 0;
        uint32_t base = 0;
        for (bool done = false; !done;)
        {
            if (base >= R.total)
            {
                row0 += per_chunk;
                done = row0 >= B.rows.n;
                if (!done)
                {
                    R = stencil_runs(F, B.gb, B.rows, g.start, row0, B.gd, lane);
                    base = 0;
                    if (R.total == 0)
                        continue;
                }
            }
            if (!done)
            {
                const uint32_t t = base + static_cast<uint32_t>(lane);
                const int r = warp_run_of(R.off, t);
                const uint32_t cs = __shfl_sync(GR_FULL, R.first, r) + t;
                const int wr = __shfl_sync(GR_FULL, R.wrap, r);
                bool keep = t < R.total;
                base += 32;
                float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
                if (keep)
                    c = g.cpos[cs];
                float vx = 0.f, vy = 0.f, vz = 0.f;
                if (!plain)
                {
                    // image for a query in the box: k = n_j - wrap (AABBQuery.cc:93,125)
                    const int pim = __float_as_int(c.w);
                    const int kx = img_ax(pim, 0) - (wr % 3 - 1);
                    const int ky = img_ax(pim, 1) - ((wr / 3) % 3 - 1);
                    const int kz = img_ax(pim, 2) - (wr / 9 - 1);
                    vx = static_cast<float>(kx);
                    vy = static_cast<float>(ky);
                    vz = static_cast<float>(kz);
                    if (!qout)
                    {
                        keep = keep && kx >= -1 && kx <= 1 && ky >= -1 && ky <= 1 && kz >= -1 && kz <= 1;
                        const float* iv = box.img[keep ? 13 - kx * 9 - ky * 3 - kz : 13]; // of -k: negated
                        vx = iv[0];
                        vy = iv[1];
                        vz = iv[2];
                    }
                }
                if (!qout)
                    keep = keep && group_gap2(B.gd, c.x + vx, c.y + vy, c.z + vz) <= cull2;
                const unsigned m = __ballot_sync(GR_FULL, keep);
                if (keep)
                {
                    const uint32_t e = n + __popc(m & lt);
                    B.x[e] = c.x;
                    B.y[e] = c.y;
                    B.z[e] = c.z;
                    B.s[e] = cs + 1;
                    if (!plain)
                    {
                        B.vx[e] = vx;
                        B.vy[e] = vy;
                        B.vz[e] = vz;
                    }
                }
                n += __popc(m);
            }
            if (n <= QB_CAP - 32 && !done)
                continue;
            // ---- the buffered candidates: list each lane's bonds, then sum them
            __syncwarp();
            if (lane < 3)
            {
                B.x[n + lane] = GR_FAR;
                B.s[n + lane] = 0;
                B.vx[n + lane] = 0.0f;
            }
            __syncwarp();
            // squared distance of candidate e to the lane's query in the pair arithmetic of
            // the ball query, with bool in: one of the reference's images
            auto image_of = [&](uint32_t e, float& ux, float& uy, float& uz) {
                // the subtrahend -(q + v), exact negations throughout
                ux = -q.x;
                uy = -q.y;
                uz = -q.z;
                if (plain)
                    return true;
                if (!qout)
                {
                    ux = __fadd_rn(ux, B.vx[e]);
                    uy = __fadd_rn(uy, B.vy[e]);
                    uz = __fadd_rn(uz, B.vz[e]);
                    return true;
                }
                const int qimg = __float_as_int(q.w);
                const float kx = B.vx[e] - static_cast<float>(img_ax(qimg, 0));
                const float ky = B.vy[e] - static_cast<float>(img_ax(qimg, 1));
                const float kz = B.vz[e] - static_cast<float>(img_ax(qimg, 2));
                const bool in = fmaxf(fmaxf(fabsf(kx), fabsf(ky)), fabsf(kz)) <= 1.0f;
                const float* v = box.img[in ? static_cast<int>(kx * 9.0f + ky * 3.0f + kz) + 13 : 13];
                ux = -__fadd_rn(q.x, v[0]);
                uy = -__fadd_rn(q.y, v[1]);
                uz = -__fadd_rn(q.z, v[2]);
                return in;
            };
            const uint32_t list0 = static_cast<uint32_t>(__cvta_generic_to_shared(&B.list[0][lane]));
            uint32_t lp = list0; // the lane's next list entry
            auto note = [&](uint32_t e, float rsq, bool in, uint32_t s) {
                if (in && rsq < p.r_max_sq && rsq >= p.r_min_sq && s != own)
                {
                    asm volatile("st.shared.u8 [%0], %1;" ::"r"(lp), "r"(e));
                    lp += 32;
                }
            };
            for (uint32_t e0 = 0; e0 < n; e0 += 32)
            {
                const uint32_t e1 = min(n, e0 + 32);
                if (!qout)
                {
                    // r = c - (q + v) = c + (-q - v), v of the candidate (plain: 0)
#pragma unroll 1
                    for (uint32_t e = e0; e < e1; e += 4)
                    {
                        const ulonglong2 cx = *reinterpret_cast<const ulonglong2*>(B.x + e);
                        const ulonglong2 cy = *reinterpret_cast<const ulonglong2*>(B.y + e);
                        const ulonglong2 cz = *reinterpret_cast<const ulonglong2*>(B.z + e);
                        const uint4 s = *reinterpret_cast<const uint4*>(B.s + e);
                        f32x2 ax = nqx, ay = nqy, az = nqz, bx = nqx, by = nqy, bz = nqz;
                        if (!plain)
                        {
                            const ulonglong2 vx = *reinterpret_cast<const ulonglong2*>(B.vx + e);
                            const ulonglong2 vy = *reinterpret_cast<const ulonglong2*>(B.vy + e);
                            const ulonglong2 vz = *reinterpret_cast<const ulonglong2*>(B.vz + e);
                            ax = add2(ax, vx.x);
                            ay = add2(ay, vy.x);
                            az = add2(az, vz.x);
                            bx = add2(bx, vx.y);
                            by = add2(by, vy.y);
                            bz = add2(bz, vz.y);
                        }
                        ax = add2(cx.x, ax);
                        ay = add2(cy.x, ay);
                        az = add2(cz.x, az);
                        bx = add2(cx.y, bx);
                        by = add2(cy.y, by);
                        bz = add2(cz.y, bz);
                        const f32x2 ra = add2(add2(fma2(ax, ax, nz), fma2(ay, ay, nz)), fma2(az, az, nz));
                        const f32x2 rb = add2(add2(fma2(bx, bx, nz), fma2(by, by, nz)), fma2(bz, bz, nz));
                        float r0, r1, r2, r3;
                        unpack2(ra, r0, r1);
                        unpack2(rb, r2, r3);
                        note(e, r0, true, s.x);
                        note(e + 1, r1, true, s.y);
                        note(e + 2, r2, true, s.z);
                        note(e + 3, r3, true, s.w);
                    }
                }
                else
                {
#pragma unroll 1
                    for (uint32_t e = e0; e < e1; ++e)
                    {
                        float ux, uy, uz;
                        const bool in = image_of(e, ux, uy, uz);
                        note(e, dot3(__fadd_rn(B.x[e], ux), __fadd_rn(B.y[e], uy), __fadd_rn(B.z[e], uz)), in, B.s[e]);
                    }
                }
                const uint32_t cnt = (lp - list0) / 32;
                if (e1 < n && !__any_sync(GR_FULL, cnt > Q_ROWS - 32))
                    continue;
                // ---- sum the listed bonds, two at a time
                __syncwarp();
                const uint32_t most = __reduce_max_sync(GR_FULL, cnt);
                for (uint32_t k = 0; k < most; k += 2)
                {
                    if (k < cnt)
                    {
                        const uint32_t ea = B.list[k][lane];
                        const bool on1 = k + 1 < cnt;
                        const uint32_t eb = on1 ? B.list[k + 1][lane] : ea;
                        const f32x2 dx = add2(pack2(B.x[ea], B.x[eb]), nqx), dy = add2(pack2(B.y[ea], B.y[eb]), nqy),
                                    dz = add2(pack2(B.z[ea], B.z[eb]), nqz);
                        f32x2 wx, wy, wz;
                        float r0, r1;
                        if (plain && !box.tilted)
                        {
                            wx = wrap_axis2<true>(box, 0, dx, nz);
                            wy = wrap_axis2<true>(box, 1, dy, nz);
                            wz = box.is2d ? 0ull : wrap_axis2<true>(box, 2, dz, nz);
                            unpack2(add2(add2(fma2(dx, dx, nz), fma2(dy, dy, nz)), fma2(dz, dz, nz)), r0, r1);
                        }
                        else if (in_box && !box.tilted)
                        {
                            wx = wrap_axis2<false>(box, 0, dx, nz);
                            wy = wrap_axis2<false>(box, 1, dy, nz);
                            wz = box.is2d ? 0ull : wrap_axis2<false>(box, 2, dz, nz);
                            const f32x2 rx = add2(pack2(B.x[ea], B.x[eb]), add2(nqx, pack2(B.vx[ea], B.vx[eb])));
                            const f32x2 ry = add2(pack2(B.y[ea], B.y[eb]), add2(nqy, pack2(B.vy[ea], B.vy[eb])));
                            const f32x2 rz = add2(pack2(B.z[ea], B.z[eb]), add2(nqz, pack2(B.vz[ea], B.vz[eb])));
                            unpack2(add2(add2(fma2(rx, rx, nz), fma2(ry, ry, nz)), fma2(rz, rz, nz)), r0, r1);
                        }
                        else
                        {
                            float a[3], b[3], ux, uy, uz;
                            image_of(ea, ux, uy, uz);
                            r0 = dot3(__fadd_rn(B.x[ea], ux), __fadd_rn(B.y[ea], uy), __fadd_rn(B.z[ea], uz));
                            image_of(eb, ux, uy, uz);
                            r1 = dot3(__fadd_rn(B.x[eb], ux), __fadd_rn(B.y[eb], uy), __fadd_rn(B.z[eb], uz));
                            float x0, x1, y0, y1, z0, z1;
                            unpack2(dx, x0, x1);
                            unpack2(dy, y0, y1);
                            unpack2(dz, z0, z1);
                            box_wrap(box, x0, y0, z0, a[0], a[1], a[2]);
                            box_wrap(box, x1, y1, z1, b[0], b[1], b[2]);
                            wx = pack2(a[0], b[0]);
                            wy = pack2(a[1], b[1]);
                            wz = pack2(a[2], b[2]);
                        }
                        add_harmonics<L>(acc, wx, wy, wz, r0, r1, on1);
                    }
                }
                bonds += cnt;
                if (LIST && most > 0)
                {
                    const uint32_t size = SEG_HEAD + 32 * most;
                    if (cend - cur < size)
                    {
                        const unsigned long long want = size > SEG_CHUNK ? size : SEG_CHUNK;
                        unsigned long long b0 = 0;
                        if (lane == 0)
                            b0 = atomicAdd(alloc, want);
                        cur = __shfl_sync(GR_FULL, b0, 0);
                        cend = cur + want;
                    }
                    if (cur + size <= cap) // past cap: the caller runs it again with room
                    {
                        uint32_t* const S = segs + cur;
                        S[lane] = cnt;
                        S[32 + lane] = slot;
                        if (lane == 0)
                        {
                            S[64] = 0;
                            *(prev_next == 0 ? head + id : segs + (prev_next - 1)) = static_cast<uint32_t>(cur) + 1;
                        }
                        prev_next = static_cast<uint32_t>(cur) + 64 + 1;
                        for (uint32_t k = 0; k < most; ++k)
                            S[SEG_HEAD + 32 * k + lane] = k < cnt ? B.s[B.list[k][lane]] - 1 : 0u;
                    }
                    cur += size;
                }
                lp = list0;
                __syncwarp();
            }
            n = 0;
            __syncwarp();
        }
        // ---- the particles' rows: q_lm = sum / bonds, through shared memory
        if (L > 0)
            acc[1] = 0ull;
        float* const tr = B.x; // [32][2 L + 3]: odd stride, no bank conflicts
        constexpr int TS = 2 * (L + 1) + 1;
        static_assert(32 * TS <= 6 * QB_N, "the rows fit the candidate arrays");
        const bool live = static_cast<uint32_t>(lane) < it.w;
        float part = 0.0f;
        {
            const float inv = 1.0f / static_cast<float>(bonds);
#pragma unroll
            for (int v = 0; v < 2 * (L + 1); ++v)
            {
                float a, b;
                unpack2(acc[v], a, b);
                const float x = (a + b) * inv;
                tr[lane * TS + v] = v == 1 ? 0.0f : x;
                if (v != 1)
                    part += (v < 2 ? 1.0f : 2.0f) * (x * x);
            }
            if (bonds == 0)
                tr[lane * TS + 1] = __int_as_float(0x7fffffff);
        }
        uint32_t i = 0;
        if (live)
        {
            i = g.cidx[slot];
            ql[static_cast<size_t>(i) * nl + k_out] = sqrtf(part * norm);
        }
        B.s[lane] = i; // (past the rows: the slots' array is not read any more)
        B.s[32 + lane] = slot;
        __syncwarp();
        constexpr uint32_t W = 2 * L + 1;
        for (uint32_t t = lane; t < it.w * W; t += 32)
        {
            const uint32_t w = t / W;
            const int c = static_cast<int>(t - w * W);
            const int m = c <= L ? c : c - L;
            float re = tr[w * TS + 2 * m], im = tr[w * TS + 2 * m + 1];
            if (c > L) // Y_l^{-m} = (-1)^m conj(Y_l^m)
            {
                re = (m & 1) ? -re : re;
                im = (m & 1) ? im : -im;
            }
            qlm[static_cast<size_t>(B.s[w]) * W + c] = make_float2(re, im);
        }
        constexpr uint32_t H = RS / 2;
        for (uint32_t t = lane; t < it.w * H; t += 32)
        {
            const uint32_t w = t / H;
            const uint32_t c = t - w * H;
            const float2 v = c <= L ? make_float2(tr[w * TS + 2 * c], tr[w * TS + 2 * c + 1]) : make_float2(0.f, 0.f);
            reinterpret_cast<float2*>(rows_out + static_cast<size_t>(B.s[32 + w]) * RS)[c] = v;
        }
        __syncwarp();
    }
}

// Neighbour averaging (Steinhardt.cc:224-289) over the groups' bond lists: a warp per
// group, P lanes per particle, lane t of them the row's floats 4 t .. 4 t + 3 (two
// orders); ave = (sum of the neighbours' rows + the own row) / (bonds + 1). Rows are the
// compact rows in slot order, so a group's neighbours lie in a few runs of memory and
// come from L1 or L2. Bound by the latency of the row loads: eight rows of 16 bytes a
// lane in flight and eight (l <= 7) particles at a time.
constexpr int AW = 8; // warps per block

template<int L>
__global__ void __launch_bounds__(AW * 32)
    k_frames_ave(const uint4* __restrict__ items, const uint32_t* __restrict__ n_items,
                 const uint32_t* __restrict__ head, const uint32_t* __restrict__ segs,
                 const uint32_t* __restrict__ cidx, BatchGrid g, const float* __restrict__ rows,
                 float* __restrict__ rows_ave, float norm, int nl, int k_out, float* __restrict__ ql_ave)
{
    constexpr int R4 = row_floats(L) / 4; // row in float4
    constexpr int P = R4 <= 1 ? 1 : (R4 <= 2 ? 2 : (R4 <= 4 ? 4 : 8));
    constexpr int PER = 32 / P;
    const float4* const rows4 = reinterpret_cast<const float4*>(rows);
    const int lane = threadIdx.x & 31;
    const int sub = lane % P;
    const bool on = sub < R4;
    const uint32_t total = *n_items;
    for (uint32_t id = blockIdx.x * AW + (threadIdx.x >> 5); id < total; id += gridDim.x * AW)
    {
        const uint4 it = items[id];
        const uint32_t first = head[id];
        uint32_t slot = 0;
        if (first == 0)
        {
            // no bonds at all: the group's slots are in no segment
            const FrameDesc& F = g.fd[it.x];
            slot = group_slot(F, group_box(F, it.y), g.start, it.z, lane);
        }
        else
        {
            slot = segs[first - 1 + 32 + lane];
        }
        const uint32_t point = static_cast<uint32_t>(lane) < it.w ? cidx[slot] : 0u;
        for (uint32_t w0 = 0; w0 < it.w; w0 += PER)
        {
            const uint32_t w = w0 + lane / P;
            const uint32_t sw = __shfl_sync(GR_FULL, slot, w & 31u), pw = __shfl_sync(GR_FULL, point, w & 31u);
            const bool live = w < it.w;
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), own = sum;
            if (live && on)
                own = rows4[static_cast<size_t>(sw) * R4 + sub];
            uint32_t count = 0;
            for (uint32_t at = first; at != 0;)
            {
                const uint32_t* S = segs + (at - 1);
                const uint32_t c = live ? S[w] : 0u;
                const uint32_t* nb = S + SEG_HEAD + w;
                at = S[64];
                for (uint32_t k = 0; k < c; k += 8)
                {
                    uint32_t j[8];
                    float4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        j[u] = k + u < c ? nb[32 * (k + u)] : 0u;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = on && k + u < c ? rows4[static_cast<size_t>(j[u]) * R4 + sub]
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                    {
                        sum.x += v[u].x;
                        sum.y += v[u].y;
                        sum.z += v[u].z;
                        sum.w += v[u].w;
                    }
                }
                count += c;
            }
            float part = 0.0f;
            if (live && on)
            {
                const float inv = 1.0f / static_cast<float>(count + 1u);
                const float4 q = make_float4((sum.x + own.x) * inv, (sum.y + own.y) * inv, (sum.z + own.z) * inv,
                                             (sum.w + own.w) * inv);
                reinterpret_cast<float4*>(rows_ave)[static_cast<size_t>(sw) * R4 + sub] = q;
                // |q_l0|^2 + 2 sum |q_lm|^2 (the padding is zero)
                part = (sub == 0 ? 1.0f : 2.0f) * (q.x * q.x + q.y * q.y);
                if (2 * sub + 1 <= L)
                    part += 2.0f * (q.z * q.z + q.w * q.w);
            }
#pragma unroll
            for (int o = P / 2; o > 0; o >>= 1)
                part += __shfl_xor_sync(GR_FULL, part, o, P);
            if (live && sub == 0)
                ql_ave[static_cast<size_t>(pw) * nl + k_out] = sqrtf(part * norm);
        }
    }
}

// hi + lo += v with the rounding error of hi + v kept exactly (TwoSum).
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float v)
{
    const float s = __fadd_rn(hi, v);
    const float bp = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(v, bp));
    hi = s;
    lo = __fadd_rn(lo, err);
}

// System sums of one split of a frame's compact rows (a frame's slots are consecutive):
// thread t takes order t mod (l + 1) of every (256 div (l + 1))-th row, float-float
// running sums, then the columns' threads in FP64 in a fixed order, as k_frames_sys.
// partial[f][split] is the l's columns in the order 0 .. l, -1 .. -l at stride, col0.
__global__ void __launch_bounds__(256)
    k_rows_sys(const uint32_t* __restrict__ pt_base, int l, int rs, int stride, int col0, int splits,
               const float* __restrict__ rows, double* __restrict__ partial)
{
    __shared__ double s_re[256];
    __shared__ double s_im[256];
    const uint32_t f = blockIdx.x, split = blockIdx.y;
    const uint32_t r_lo = pt_base[f];
    const uint32_t nf = pt_base[f + 1] - r_lo;
    const uint32_t per = (nf + splits - 1) / splits;
    const uint32_t r0 = r_lo + min(nf, split * per);
    const uint32_t r1 = r_lo + min(nf, (split + 1) * per);
    const int t = threadIdx.x;
    const int nm = l + 1, per_pass = 256 / nm;
    const int m = t % nm, rr = t / nm;
    float hr = 0.f, lr = 0.f, hi = 0.f, li = 0.f;
    if (rr < per_pass)
    {
        for (uint32_t r = r0 + rr; r < r1; r += per_pass)
        {
            const float2 v = reinterpret_cast<const float2*>(rows + static_cast<size_t>(r) * rs)[m];
            two_sum_acc(hr, lr, v.x);
            two_sum_acc(hi, li, v.y);
        }
    }
    s_re[t] = static_cast<double>(hr) + static_cast<double>(lr);
    s_im[t] = static_cast<double>(hi) + static_cast<double>(li);
    __syncthreads();
    if (t < nm)
    {
        double ar = 0.0, ai = 0.0;
        for (int q = 0; q < per_pass; ++q)
        {
            ar += s_re[q * nm + t];
            ai += s_im[q * nm + t];
        }
        double* out = partial + ((static_cast<size_t>(f) * splits + split) * stride + col0) * 2;
        out[2 * t] = ar;
        out[2 * t + 1] = ai;
        if (t > 0)
        {
            out[2 * (l + t)] = (t & 1) ? -ar : ar;
            out[2 * (l + t) + 1] = (t & 1) ? ai : -ai;
        }
    }
}

// ---- small systems without tilt, no grid -------------------------------------------------
// A warp per particle: 32 points at a time are tested (the nearest image as in the small
// histogram), the bonds listed, and then taken two a lane; the lanes' sums meet by shuffles.
// Less than the latency of a grid and of groups whose lanes walk their bonds one after the
// other: whole calls of l = 6 at density 1, r_max 1.2 to 3, 1000 points 98 to 101 us against 128 to
// 326 by groups, 3000 137 to 141 / 141 to 320, 5000 206 to 217 / 160 to 323; averaged, r_max 1.2 to 2, 116
// to 121 / 162 to 234, 153 to 156 / 171 to 281, 222 to 231 / 199 to 293. (fg_capi.cu has the rule.)
constexpr int SQ_WARPS = 4;
constexpr int SQ_LIST = 128; // listed bonds a warp

template<int L>
__global__ void __launch_bounds__(SQ_WARPS * 32)
    k_small_qlm(DevBox b, const float* __restrict__ pts, uint32_t n, BallParams p, float norm, int nl, int k_out,
                float2* __restrict__ qlm, float* __restrict__ ql, float* __restrict__ rows_out,
                uint32_t* __restrict__ nb, uint32_t* __restrict__ nb_count)
{
    constexpr int RS = row_floats(L);
    constexpr int W = 2 * L + 1;
    __shared__ uint2 s_list[SQ_WARPS][SQ_LIST]; // point, r^2
    __shared__ float s_row[SQ_WARPS][32];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t i = blockIdx.x * SQ_WARPS + warp;
    if (i >= n)
        return;
    uint2* const list = s_list[warp];
    const float* const pi = pts + 3 * static_cast<size_t>(i);
    const float q[3] = {pi[0], pi[1], b.is2d ? 0.0f : pi[2]};
    const float up[3] = {__fadd_rn(q[0], b.img[22][0]), __fadd_rn(q[1], b.img[16][1]), __fadd_rn(q[2], b.img[14][2])};
    const float dn[3] = {__fadd_rn(q[0], b.img[4][0]), __fadd_rn(q[1], b.img[10][1]), __fadd_rn(q[2], b.img[12][2])};
    auto axis = [](float x, float q0, float q1, float q2) {
        return fminf(fminf(fabsf(__fsub_rn(x, q0)), fabsf(__fsub_rn(x, q1))), fabsf(__fsub_rn(x, q2)));
    };
    f32x2 acc[2 * (L + 1)];
#pragma unroll
    for (int v = 0; v < 2 * (L + 1); ++v)
        acc[v] = 0ull;
    uint32_t cnt = 0, bonds = 0;
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < n || cnt > 0; j0 += 32)
    {
        if (j0 < n)
        {
            const uint32_t j = j0 + lane;
            bool ok = false;
            float rsq = 0.0f;
            if (j < n)
            {
                const float* pj = pts + 3 * static_cast<size_t>(j);
                rsq = dot3(axis(pj[0], q[0], up[0], dn[0]), axis(pj[1], q[1], up[1], dn[1]),
                           axis(b.is2d ? 0.0f : pj[2], q[2], up[2], dn[2]));
                ok = rsq < p.r_max_sq && rsq >= p.r_min_sq && !(p.exclude_ii && j == i);
            }
            const unsigned m = __ballot_sync(GR_FULL, ok);
            if (ok)
            {
                const uint32_t at = __popc(m & lt);
                list[cnt + at] = make_uint2(j, __float_as_uint(rsq));
                if (nb != nullptr && bonds + at < SMALL_ST_BONDS)
                    nb[static_cast<size_t>(i) * SMALL_ST_BONDS + bonds + at] = j;
            }
            cnt += __popc(m);
            bonds += __popc(m);
        }
        if (cnt <= SQ_LIST - 32 && j0 + 32 < n)
            continue;
        __syncwarp();
#pragma unroll 1
        for (uint32_t e = lane; e < cnt; e += 64)
        {
            const bool on1 = e + 32 < cnt;
            const uint2 a = list[e], c = list[on1 ? e + 32 : e];
            float x[3], y[3];
            const float* pa = pts + 3 * static_cast<size_t>(a.x);
            const float* pc = pts + 3 * static_cast<size_t>(c.x);
            box_wrap(b, __fsub_rn(pa[0], q[0]), __fsub_rn(pa[1], q[1]), __fsub_rn(b.is2d ? 0.0f : pa[2], q[2]), x[0], x[1],
                     x[2]);
            box_wrap(b, __fsub_rn(pc[0], q[0]), __fsub_rn(pc[1], q[1]), __fsub_rn(b.is2d ? 0.0f : pc[2], q[2]), y[0], y[1],
                     y[2]);
            add_harmonics<L>(acc, pack2(x[0], y[0]), pack2(x[1], y[1]), pack2(x[2], y[2]), __uint_as_float(a.y),
                             __uint_as_float(c.y), on1);
        }
        cnt = 0;
        __syncwarp();
    }
    if (L > 0)
        acc[1] = 0ull;
    s_row[warp][lane] = 0.0f;
    __syncwarp();
    const float inv = 1.0f / static_cast<float>(bonds);
    float part = 0.0f;
#pragma unroll
    for (int v = 0; v < 2 * (L + 1); ++v)
    {
        float x, y;
        unpack2(acc[v], x, y);
        x += y;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            x += __shfl_xor_sync(GR_FULL, x, o);
        x *= inv;
        if (v != 1)
            part += (v < 2 ? 1.0f : 2.0f) * (x * x);
        if (lane == 0)
            s_row[warp][v] = v == 1 ? (bonds == 0 ? __int_as_float(0x7fffffff) : 0.0f) : x;
    }
    __syncwarp();
    if (lane == 0)
    {
        ql[static_cast<size_t>(i) * nl + k_out] = sqrtf(part * norm);
        if (nb_count != nullptr)
            nb_count[i] = bonds;
    }
    if (lane < W)
    {
        const int m = lane <= L ? lane : lane - L;
        float re = s_row[warp][2 * m], im = s_row[warp][2 * m + 1];
        if (lane > L) // Y_l^{-m} = (-1)^m conj(Y_l^m)
        {
            re = (m & 1) ? -re : re;
            im = (m & 1) ? im : -im;
        }
        qlm[static_cast<size_t>(i) * W + lane] = make_float2(re, im);
    }
    if (lane < RS)
        rows_out[static_cast<size_t>(i) * RS + lane] = s_row[warp][lane];
}

// Neighbour averaging over the listed neighbours: a warp per particle, a lane per float of
// the row. *over: some particle has more neighbours than are listed.
template<int L>
__global__ void __launch_bounds__(SQ_WARPS * 32)
    k_small_ave(uint32_t n, const uint32_t* __restrict__ nb, const uint32_t* __restrict__ nb_count,
                const float* __restrict__ rows, float* __restrict__ rows_ave, float norm, int nl, int k_out,
                float* __restrict__ ql_ave, int* __restrict__ over)
{
    constexpr int RS = row_floats(L);
    const int lane = threadIdx.x & 31;
    const uint32_t i = blockIdx.x * SQ_WARPS + (threadIdx.x >> 5);
    if (i >= n)
        return;
    const uint32_t count = nb_count[i];
    if (count > SMALL_ST_BONDS)
    {
        if (lane == 0)
            atomicOr(over, 1);
        return;
    }
    const uint32_t* const list = nb + static_cast<size_t>(i) * SMALL_ST_BONDS;
    const int c = min(lane, RS - 1);
    float sum = 0.0f;
#pragma unroll 8
    for (uint32_t e = 0; e < count; ++e)
        sum += rows[static_cast<size_t>(list[e]) * RS + c];
    const float x = (sum + rows[static_cast<size_t>(i) * RS + c]) * (1.0f / static_cast<float>(count + 1u));
    float part = lane < 2 * (L + 1) ? (lane < 2 ? 1.0f : 2.0f) * (x * x) : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        part += __shfl_xor_sync(GR_FULL, part, o);
    if (lane == 0)
        ql_ave[static_cast<size_t>(i) * nl + k_out] = sqrtf(part * norm);
    if (lane < RS)
        rows_ave[static_cast<size_t>(i) * RS + lane] = x;
}

// System sums of n compact rows of one l over n, by one block: float-float running sums, then
// FP64 in a fixed order, as k_rows_sys and k_frames_sys_final.
constexpr int SS_T = 512;
__global__ void __launch_bounds__(SS_T)
    k_small_sys(uint32_t n, int l, int rs, const float* __restrict__ rows, double* __restrict__ sys)
{
    __shared__ double s_re[SS_T];
    __shared__ double s_im[SS_T];
    const int t = threadIdx.x;
    const int nm = l + 1, per_pass = SS_T / nm;
    const int m = t % nm, rr = t / nm;
    float hr = 0.f, lr = 0.f, hi = 0.f, li = 0.f;
    if (rr < per_pass)
    {
#pragma unroll 8
        for (uint32_t r = rr; r < n; r += per_pass)
        {
            const float2 v = reinterpret_cast<const float2*>(rows + static_cast<size_t>(r) * rs)[m];
            two_sum_acc(hr, lr, v.x);
            two_sum_acc(hi, li, v.y);
        }
    }
    s_re[t] = static_cast<double>(hr) + static_cast<double>(lr);
    s_im[t] = static_cast<double>(hi) + static_cast<double>(li);
    // a tree over the rows of a pass
    for (int half = 256; half > 0; half >>= 1)
    {
        __syncthreads();
        if (rr < half && rr + half < per_pass)
        {
            s_re[t] += s_re[t + half * nm];
            s_im[t] += s_im[t + half * nm];
        }
    }
    __syncthreads();
    if (t < nm)
    {
        const double ar = s_re[t] / n, ai = s_im[t] / n;
        sys[2 * t] = ar;
        sys[2 * t + 1] = ai;
        if (t > 0)
        {
            sys[2 * (l + t)] = (t & 1) ? -ar : ar;
            sys[2 * (l + t) + 1] = (t & 1) ? ai : -ai;
        }
    }
}

template<int L> void go_small(const SmallQlm& w, int k, cudaStream_t s)
{
    const uint32_t blocks = (w.n + SQ_WARPS - 1) / SQ_WARPS;
    {
        ProfScope prof_("k_small_qlm", s);
        k_small_qlm<L><<<blocks, SQ_WARPS * 32, 0, s>>>(w.b, w.pts, w.n, w.p, w.ls->norm[k], w.ls->nl, k,
                                                      w.qlm + w.ls->qlm_offset[k], w.ql, w.rows, k == 0 ? w.nb : nullptr,
                                                      k == 0 ? w.nb_count : nullptr);
    }
    if (w.nb != nullptr)
    {
        ProfScope prof_("k_small_ave", s);
        k_small_ave<L><<<blocks, SQ_WARPS * 32, 0, s>>>(w.n, w.nb, w.nb_count, w.rows, w.rows_ave, w.ls->norm[k], w.ls->nl,
                                                      k, w.ql_ave, w.over);
    }
}

using GoSmall = void (*)(const SmallQlm&, int, cudaStream_t);
template<int... I> GoSmall small_entry(int l, std::integer_sequence<int, I...>)
{
    static const GoSmall table[] = {go_small<I>...};
    return table[l];
}

int sm_total()
{
    static int v = 0;
    if (v == 0)
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        v = std::max(v, 1);
    }
    return v;
}

template<int L, bool LIST>
uint32_t qlm_blocks(uint32_t expected)
{
    static int per = 0;
    if (per == 0)
    {
        const int smem = static_cast<int>(sizeof(QBuf)) * QW;
        cudaFuncSetAttribute(k_frames_qlm<L, LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_frames_qlm<L, LIST>, QW * 32, smem);
        per = std::max(per, 1);
    }
    return std::min<uint32_t>(static_cast<uint32_t>(sm_total() * per), std::max<uint32_t>(1u, (expected + QW - 1) / QW));
}

template<int L>
void go_qlm(const BatchGrid& g, const BallParams& p, const FrameQlm& w, int k, cudaStream_t s)
{
    const size_t smem = sizeof(QBuf) * QW;
    if (w.list && k == 0)
    {
        ProfScope prof_("k_frames_qlm<LIST>", s);
        k_frames_qlm<L, true><<<qlm_blocks<L, true>(w.expected), QW * 32, smem, s>>>(
            g, p, NEG_ZERO2, w.items, w.n_items, w.queue + k, w.ls->norm[k], w.ls->nl, k, w.qlm + w.ls->qlm_offset[k],
            w.ql, w.rows, w.head, w.segs, w.alloc, w.cap);
    }
    else
    {
        ProfScope prof_("k_frames_qlm", s);
        k_frames_qlm<L, false><<<qlm_blocks<L, false>(w.expected), QW * 32, smem, s>>>(
            g, p, NEG_ZERO2, w.items, w.n_items, w.queue + k, w.ls->norm[k], w.ls->nl, k, w.qlm + w.ls->qlm_offset[k],
            w.ql, w.rows, nullptr, nullptr, nullptr, 0);
    }
    if (w.list)
    {
        ProfScope prof_("k_frames_ave", s);
        const uint32_t blocks = std::min<uint32_t>(static_cast<uint32_t>(sm_total()) * 8u, (w.expected + AW - 1) / AW);
        k_frames_ave<L><<<std::max(blocks, 1u), AW * 32, 0, s>>>(w.items, w.n_items, w.head, w.segs, g.cidx, g, w.rows,
                                                             w.rows_ave, w.ls->norm[k], w.ls->nl, k, w.ql_ave);
    }
}

using GoQlm = void (*)(const BatchGrid&, const BallParams&, const FrameQlm&, int, cudaStream_t);
template<int... I> GoQlm qlm_entry(int l, std::integer_sequence<int, I...>)
{
    static const GoQlm table[] = {go_qlm<I>...};
    return table[l];
}

} // namespace

int frame_row_floats(int l)
{
    return row_floats(l);
}

uint64_t frame_segment_words(double groups, double bonds_per_point, uint32_t expected)
{
    // rows of a group (a segment's head is 3): while a group's bonds are summed once, the most bonds of its 32
    // lanes, about three deviations above the mean; more bonds are summed in several sweeps, each
    // with its own most, which add up to 2.1 (30 bonds a point), 2.4 (100) to 3.0 (270) times the
    // mean of uniform points. Too few words run the call again: 1M points, 100 bonds, twice the work.
    const double once = bonds_per_point + 3.0 * std::sqrt(bonds_per_point) + 5.0;
    const double rows = bonds_per_point > 16.0 ? std::max(once, 3.1 * bonds_per_point) : once;
    const uint64_t slack = static_cast<uint64_t>(qlm_blocks<6, true>(expected)) * QW * SEG_CHUNK;
    return static_cast<uint64_t>(groups * 32.0 * rows) + slack;
}

void launch_frames_qlm(const BatchGrid& g, const BallParams& p, const FrameQlm& w, int k, cudaStream_t s)
{
    qlm_entry(w.ls->l[k], std::make_integer_sequence<int, FRAME_QLM_MAX_L + 1>())(g, p, w, k, s);
}

void launch_small_qlm(const SmallQlm& w, cudaStream_t s)
{
    int col = 0;
    for (int k = 0; k < w.ls->nl; ++k)
    {
        const int l = w.ls->l[k];
        small_entry(l, std::make_integer_sequence<int, FRAME_QLM_MAX_L + 1>())(w, k, s);
        ProfScope prof_("k_small_sys", s);
        k_small_sys<<<1, SS_T, 0, s>>>(w.n, l, row_floats(l), w.nb != nullptr ? w.rows_ave : w.rows, w.sys + 2 * col);
        col += 2 * l + 1;
    }
}

void launch_rows_sys(const uint32_t* pt_base, uint32_t nframes, uint32_t max_rows, int l, int stride, int col0,
                     const float* rows, double* partial, cudaStream_t s)
{
    const int splits = frames_sys_splits(max_rows);
    ProfScope prof_("k_rows_sys", s);
    k_rows_sys<<<dim3(nframes, splits), 256, 0, s>>>(pt_base, l, row_floats(l), stride, col0, splits, rows, partial);
}

} // namespace fg
