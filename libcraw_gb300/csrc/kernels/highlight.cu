/*
 * Highlight reconstruction (reference lib/ref/ref_highlight.c, the stage
 * the reference's tools run by default): the clipped sites of a mosaic are
 * rebuilt from their unclipped neighbours and a smooth field of the
 * scene's colour, before the debayer.
 *
 *   k_hl_level0    one texel per 2x2 quads: weighted log chroma (ln R/G,
 *                  ln B/G) of the quads, and the weight, which falls to 0
 *                  within 3 quads of a clip (the quads' clip ramps and
 *                  their 7x7 max are made in registers on the way)
 *   k_hl_pull      each coarser level the sum of its four children, to 1x1
 *   k_hl_coarse    the levels of at most kCoarseTexels, pulled and pushed
 *                  in one CTA
 *   k_hl_push      back down: each texel blended from the coarser level's
 *                  bilinear colour toward its own mean by its weight
 *   k_hl_fill      per site: u * gain, lifted where a > 0 toward the level
 *                  its neighbours' channels and the field predict; fp16
 *
 * The mosaic is read twice and the fp16 mosaic written once; the field is
 * 1/16 size. Operation order follows the reference and this file is built
 * without multiply-add contraction (the oracle's -ffp-contract=off), so
 * the only differences are the device's logf/expf against the host's.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace {

constexpr float kULo = 0.92f, kUHi = 0.98f, kEps = 1e-4f, kLogMax = 2.0f, kWSat = 1.0f;
constexpr int kDilate = 3;

/* smoothstep(kULo, kUHi, v). The quotient by Markstein's correction of the
 * product with the correctly rounded reciprocal, which rounds as the division
 * does; below kULo it is not positive and clamps to 0. A product above 1 need
 * not be near (and one that overflows must not go on as infinity). */
CRAW_DEV float smooth(float v)
{
    constexpr float c = kUHi - kULo, rc = 1.0f / c;
    const float x = v - kULo, q = fminf(x * rc, 4.0f);
    const float t = __saturatef(__fmaf_rn(__fmaf_rn(-c, q, x), rc, q));
    return t * t * (3.0f - 2.0f * t);
}

CRAW_DEV float site_u(const CRAWKHighlight &k, uint16_t raw, int s)
{
    return ((float)raw * (1.0f / 65535.0f) - k.black[s]) * k.inv_range[s];
}

CRAW_DEV float fmax0(float m, float v) { return m > v ? m : v; }   /* the reference's MAX(m, v) */

CRAW_DEV float clampf(float v, float lo, float hi)
{
    return fminf(fmaxf(v, lo), hi);
}

/* Part of the frame's quads for walking warps: strips of columns, `nx`
 * across, in segments of `seg` quad rows. */
struct HlGrid {
    int nx, seg;
};

constexpr int kWalkWarps = 4, kWalkNT = 32 * kWalkWarps;

/* Level 0 of the colour field, straight from the mosaic, by walking warps: a
 * lane owns two quad columns (a column of texels) and walks down a segment of
 * quad rows. A quad row's clip ramps qa (the largest of a quad's four; 0
 * outside the grid, which is what skipping those quads gives, all ramps being
 * >= 0) give their largest over +-kDilate along x by shuffles and along y
 * from the rows before, so that kDilate rows later a quad's weight
 * (1 - amax) min(umax, 1)^2 is known, and its log chroma is formed where the
 * weight is not 0. A texel sums its quads in the reference's order: rows,
 * then columns. kL0N lanes have outputs; two on either side are their apron.
 *
 * Bound: instruction issue (two IEEE divisions and two logarithms a quad with
 * a weight). 6000x4000: 55 us, where 32x16 tiles staged in shared memory with
 * their apron (1.6 times the quads) took 72. */
constexpr int kL0N = 28, kL0Ctas = 6;
static_assert(kDilate == 3, "two lanes of apron, a window of 7");

__global__ void __launch_bounds__(kWalkNT, kL0Ctas)
k_hl_level0(const CRAWKHighlight k, const CRAWKHighlightIO io, const HlGrid g)
{
    craw_await_previous();
    craw_let_next_start();
    const int lane = threadIdx.x & 31, wid = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    const int sx = wid % g.nx, y0 = wid / g.nx * g.seg;
    const int qw = k.width / 2, qh = k.height / 2;
    if (y0 >= qh)
        return;
    const int y1 = min(y0 + g.seg, qh);
    const int tx = sx * kL0N + lane - 2, qx = 2 * tx;        /* the lane's texel, its first quad */
    const bool in0 = qx >= 0 && qx < qw, in1 = qx >= 0 && qx + 1 < qw;
    const bool mine = lane >= 2 && lane < 2 + kL0N && tx < k.lw[0];
    /* Quad row y of the lane's quads: top rows' samples, then bottom rows'. */
    auto fetch = [&](int y) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (in0 && y >= 0 && y < qh &&
            craw_in_bounds(qx >= 0 && 2 * qx + (in1 ? 3 : 1) < k.width && 2 * y + 1 < k.height, io.err)) {
            const char *row = (const char *)io.src + (size_t)(2 * y) * io.src_pitch + (size_t)qx * 4;
            if (in1) {
                const uint2 a = __ldg(reinterpret_cast<const uint2 *>(row));
                const uint2 b = __ldg(reinterpret_cast<const uint2 *>(row + io.src_pitch));
                v = make_uint4(a.x, a.y, b.x, b.y);
            } else {
                v.x = __ldg(reinterpret_cast<const uint32_t *>(row));
                v.z = __ldg(reinterpret_cast<const uint32_t *>(row + io.src_pitch));
            }
        }
        return v;
    };
    auto levels = [&](const uint4 &v, int i, float u[4]) {
        const uint32_t p0 = i ? v.y : v.x, p1 = i ? v.w : v.z;
        u[0] = site_u(k, (uint16_t)(p0 & 0xffffu), 0);
        u[1] = site_u(k, (uint16_t)(p0 >> 16), 1);
        u[2] = site_u(k, (uint16_t)(p1 & 0xffffu), 2);
        u[3] = site_u(k, (uint16_t)(p1 >> 16), 3);
    };
    /* Of the rows before: the samples of three, and the running maxima over
     * one, two and four rows that the seven are made of. */
    uint4 raw1 = make_uint4(0u, 0u, 0u, 0u), raw2 = raw1, raw3 = raw1, next = fetch(y0 - kDilate);
    float h1[2] = { 0.0f, 0.0f }, m2a[2] = { 0.0f, 0.0f }, m2b[2] = { 0.0f, 0.0f };
    float m4a[2] = { 0.0f, 0.0f }, m4b[2] = { 0.0f, 0.0f }, m4c[2] = { 0.0f, 0.0f };
    float acc[3] = { 0.0f, 0.0f, 0.0f };
#pragma unroll 1
    for (int y = y0 - kDilate; y < y1 + kDilate; y++) {
        const uint4 raw = next;
        next = fetch(y + 1);
        float m[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float u[4];
            levels(raw, i, u);
            const float t = fmaxf(fmaxf(smooth(u[0]), smooth(u[1])), fmaxf(smooth(u[2]), smooth(u[3])));
            m[i] = (i ? in1 : in0) && y >= 0 && y < qh ? t : 0.0f;
        }
        const float p = fmaxf(m[0], m[1]);
        const float t = fmaxf(fmaxf(__shfl_up_sync(0xffffffffu, p, 1), p), __shfl_down_sync(0xffffffffu, p, 1));
        const float h[2] = { fmaxf(t, __shfl_up_sync(0xffffffffu, m[1], 2)),
                             fmaxf(t, __shfl_down_sync(0xffffffffu, m[0], 2)) };
        const int r = y - kDilate;
        float amax[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float m2 = fmaxf(h[i], h1[i]), m4 = fmaxf(m2, m2b[i]);
            amax[i] = fmaxf(m4, m4c[i]);         /* rows y - 6 .. y */
            h1[i] = h[i];
            m2b[i] = m2a[i];
            m2a[i] = m2;
            m4c[i] = m4b[i];
            m4b[i] = m4a[i];
            m4a[i] = m4;
        }
        if (r >= y0) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                float u[4];
                levels(raw3, i, u);
                float umax = 0.0f;
#pragma unroll
                for (int s = 0; s < 4; s++)
                    umax = fmaxf(umax, u[s]);
                const float w = umax < 1.0f ? umax : 1.0f;
                const float wq = mine && (i ? in1 : in0) ? (1.0f - amax[i]) * w * w : 0.0f;
                /* At weight 0 the products are +-0 (the logs are clamped, so
                 * finite) and add nothing to a sum that is never -0. */
                if (wq != 0.0f) {
                    const float g0 = (u[1] * k.wb[1] + u[2] * k.wb[1]) * 0.5f, gg = fmax0(g0, kEps);
                    const float lr = clampf(logf(__fdiv_rn(fmax0(u[0] * k.wb[0], kEps), gg)), -kLogMax, kLogMax);
                    const float lb = clampf(logf(__fdiv_rn(fmax0(u[3] * k.wb[2], kEps), gg)), -kLogMax, kLogMax);
                    acc[0] += wq * lr;
                    acc[1] += wq * lb;
                    acc[2] += wq;
                }
            }
            if ((r & 1) || r == qh - 1) {
                if (mine && craw_in_bounds(tx >= 0 && tx < k.lw[0] && (r >> 1) < k.lh[0], io.err))
                    reinterpret_cast<float4 *>(io.levels)[k.off[0] + (size_t)(r >> 1) * k.lw[0] + tx] =
                        make_float4(acc[0], acc[1], acc[2], 0.0f);
                acc[0] = acc[1] = acc[2] = 0.0f;
            }
        }
        raw3 = raw2;
        raw2 = raw1;
        raw1 = raw;
    }
}

/* Texel (x, y) of level l + 1 as the sum of its children in level l. */
CRAW_DEV void pull_texel(const CRAWKHighlight &k, const CRAWKHighlightIO &io, int l, int x, int y)
{
    const int fw = k.lw[l], fh = k.lh[l];
    const float4 *f = reinterpret_cast<const float4 *>(io.levels) + k.off[l];
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
    for (int dy = 0; dy < 2; dy++)
        for (int dx = 0; dx < 2; dx++) {
            const int fx = 2 * x + dx, fy = 2 * y + dy;
            if (fx >= fw || fy >= fh)
                continue;
            const float4 t = f[(size_t)fy * fw + fx];
            a0 += t.x;
            a1 += t.y;
            a2 += t.z;
        }
    reinterpret_cast<float4 *>(io.levels)[k.off[l + 1] + (size_t)y * k.lw[l + 1] + x] =
        make_float4(a0, a1, a2, 0.0f);
}

__global__ void k_hl_pull(const CRAWKHighlight k, const CRAWKHighlightIO io, int l)
{
    craw_await_previous();
    craw_let_next_start();
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x < k.lw[l + 1] && y < k.lh[l + 1])
        pull_texel(k, io, l, x, y);
}

/* A level's colour at a texel clamped to its edge; the top level still
 * holds sums (reference ref_highlight.c:57-70). */
CRAW_DEV void texel(const float4 *t, int w, int h, int x, int y, bool top, float out[2])
{
    x = x < 0 ? 0 : (x >= w ? w - 1 : x);
    y = y < 0 ? 0 : (y >= h ? h - 1 : y);
    const float4 v = t[(size_t)y * w + x];
    if (top) {
        out[0] = v.z > 0.0f ? __fdiv_rn(v.x, v.z) : 0.0f;
        out[1] = v.z > 0.0f ? __fdiv_rn(v.y, v.z) : 0.0f;
    } else {
        out[0] = v.x;
        out[1] = v.y;
    }
}

/* Bilinear at (px, py), mixed along x first (ref_highlight.c:74-93). */
CRAW_DEV void bilinear(const float4 *t, int w, int h, float px, float py, bool top, float out[2])
{
    const float fx0 = floorf(px), fy0 = floorf(py), fx = px - fx0, fy = py - fy0;
    const int x0 = (int)fx0, y0 = (int)fy0;
    float c00[2], c10[2], c01[2], c11[2];
    texel(t, w, h, x0, y0, top, c00);
    texel(t, w, h, x0 + 1, y0, top, c10);
    texel(t, w, h, x0, y0 + 1, top, c01);
    texel(t, w, h, x0 + 1, y0 + 1, top, c11);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float a = __fadd_rn(__fmul_rn(c00[i], 1.0f - fx), __fmul_rn(c10[i], fx));
        const float b = __fadd_rn(__fmul_rn(c01[i], 1.0f - fx), __fmul_rn(c11[i], fx));
        out[i] = __fadd_rn(__fmul_rn(a, 1.0f - fy), __fmul_rn(b, fy));
    }
}

/* Texel (x, y) of level l pushed from level l + 1, in place. */
CRAW_DEV void push_texel(const CRAWKHighlight &k, const CRAWKHighlightIO &io, int l, int x, int y)
{
    const int w = k.lw[l];
    const float4 *c = reinterpret_cast<const float4 *>(io.levels) + k.off[l + 1];
    float4 *f = reinterpret_cast<float4 *>(io.levels) + k.off[l];
    float up[2];
    bilinear(c, k.lw[l + 1], k.lh[l + 1], ((float)x + 0.5f) * 0.5f - 0.5f,
             ((float)y + 0.5f) * 0.5f - 0.5f, l + 2 == k.nb_levels, up);
    float4 t = f[(size_t)y * w + x];
    if (t.z > 0.0f) {
        const float q = __fdiv_rn(t.z, kWSat), s = q < 1.0f ? q : 1.0f;
        t.x = up[0] + s * (__fdiv_rn(t.x, t.z) - up[0]);
        t.y = up[1] + s * (__fdiv_rn(t.y, t.z) - up[1]);
    } else {
        t.x = up[0];
        t.y = up[1];
    }
    f[(size_t)y * w + x] = t;
}

__global__ void k_hl_push(const CRAWKHighlight k, const CRAWKHighlightIO io, int l)
{
    craw_await_previous();
    craw_let_next_start();
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x < k.lw[l] && y < k.lh[l])
        push_texel(k, io, l, x, y);
}

/* The coarse end of the pyramid in one CTA: pull from level l0 to the top,
 * then push back down to l0, a barrier between levels (a dozen tiny
 * launches otherwise). */
constexpr int kCoarseThreads = 1024, kCoarseTexels = 8192;

__global__ void __launch_bounds__(kCoarseThreads) k_hl_coarse(const CRAWKHighlight k, const CRAWKHighlightIO io, int l0)
{
    craw_await_previous();
    craw_let_next_start();
    for (int l = l0; l + 1 < k.nb_levels; l++) {
        const int w = k.lw[l + 1], n = w * k.lh[l + 1];
        for (int i = threadIdx.x; i < n; i += kCoarseThreads)
            pull_texel(k, io, l, i % w, i / w);
        __syncthreads();
    }
    for (int l = k.nb_levels - 2; l >= l0; l--) {
        const int w = k.lw[l], n = w * k.lh[l];
        for (int i = threadIdx.x; i < n; i += kCoarseThreads)
            push_texel(k, io, l, i % w, i / w);
        __syncthreads();
    }
}

/* The lift of one site (reference ref_highlight.c:286-327): `xc` its
 * balanced value, `a` its ramp; (s1, n1, m1) and (s2, n2, m2) the sum,
 * count and largest ramp of its neighbours of the other two channels
 * k1 < k2, `rho1`, `rho2`, `rhoc` their and its own log chroma. The
 * counts are 2 or 4, so the means are products with 1/n, which round as
 * the quotients do. */
CRAW_DEV float lift(float xc, float a, float s1, float inv_n1, float m1, float s2, float inv_n2, float m2,
                    float rho1, float rho2, float rhoc)
{
    const float a1 = 1.0f - m1, a2 = 1.0f - m2;
    const float l1 = logf(fmax0(s1 * inv_n1, kEps)) - rho1;
    const float l2 = logf(fmax0(s2 * inv_n2, kEps)) - rho2;
    const float lc = logf(fmax0(xc, kEps)) - rhoc;
    const float A = a1 + a2;
    const float lfull = expf(fmax0(lc, fmax0(l1, l2)));
    float L = lfull;
    if (A > 0.0f) {
        const float lpart = expf(__fdiv_rn(a1 * l1 + a2 * l2, A));
        L = lfull + (A < 1.0f ? A : 1.0f) * (lpart - lfull);
    }
    return xc + a * fmax0(L * expf(rhoc) - xc, 0.0f);
}

/* The mirror of a row: one reflection, which is exact for the rows a window
 * reads (at most one outside the frame), then a clamp that keeps the rows no
 * window reads inside it. */
CRAW_DEV int edge(int v, int n)
{
    v = v < 0 ? -v : v;
    v = v >= n ? 2 * n - 2 - v : v;
    return v < 0 ? 0 : v;
}

/* One row of a quad's 4x4 window: u and the ramp of its own pair of samples
 * (cells 1 and 2) and of the neighbours' (0 and 3), mirrored at the frame's
 * edge (mirroring keeps parity). */
struct HlRow {
    float u[4], a[4];
};

/* The rebuilt mosaic by walking warps: a lane owns a quad column and walks
 * down a segment of quad rows, a lane of apron on either side; the 4x4 window
 * of the quad (cell (r, c) = frame position (x0 - 1 + c, y0 - 1 + r), CFA
 * site ((r + 1) & 1) * 2 + ((c + 1) & 1)) stays in its registers. A quad none
 * of whose sites is near the clip only scales its four samples; otherwise
 * each site whose ramp is above 0 is lifted. Neighbours of each channel are
 * summed in the reference's scan order (rows, then columns).
 *
 * Bound: instruction issue, the lifts' logarithms and exponentials above all
 * where a frame is clipped: so short segments, which the hardware hands out
 * as CTAs end (one wave of 67 rows each took 152 us, 16 rows 113). 6000x4000,
 * most of it clipped: 105 us, where tiles staged in shared memory took 126.
 * A small frame's time is its segment's chain of rows: fill_rows(). */
constexpr int kFillN = 30, kFillCtas = 7, kFillMost = 8, kFillWaves = 5;

__global__ void __launch_bounds__(kWalkNT, kFillCtas)
k_hl_fill(const CRAWKHighlight k, const CRAWKHighlightIO io, const HlGrid g)
{
    craw_await_previous();
    craw_let_next_start();
    const int lane = threadIdx.x & 31, wid = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    const int sx = wid % g.nx, q0 = wid / g.nx * g.seg;
    const int qw = k.width / 2, qh = k.height / 2;
    if (q0 >= qh)
        return;
    const int q1 = min(q0 + g.seg, qh), qx = sx * kFillN + lane - 1, x0 = 2 * qx;
    const bool in = qx >= 0 && qx < qw, mine = in && lane >= 1 && lane <= kFillN;
    const bool first = qx == 0, last = qx == qw - 1;
    auto fetch = [&](int y) {
        const int yr = edge(y, k.height);
        if (!in || !craw_in_bounds(yr >= 0 && yr < k.height, io.err))
            return 0u;
        return __ldg(reinterpret_cast<const uint32_t *>((const char *)io.src + (size_t)yr * io.src_pitch) + qx);
    };
    auto row = [&](uint32_t raw, int odd) {
        HlRow r;
        r.u[1] = site_u(k, (uint16_t)(raw & 0xffffu), 2 * odd);
        r.u[2] = site_u(k, (uint16_t)(raw >> 16), 2 * odd + 1);
        r.a[1] = smooth(r.u[1]);
        r.a[2] = smooth(r.u[2]);
        const float ul = __shfl_up_sync(0xffffffffu, r.u[2], 1), ur = __shfl_down_sync(0xffffffffu, r.u[1], 1);
        const float al = __shfl_up_sync(0xffffffffu, r.a[2], 1), ar = __shfl_down_sync(0xffffffffu, r.a[1], 1);
        r.u[0] = first ? r.u[2] : ul;
        r.a[0] = first ? r.a[2] : al;
        r.u[3] = last ? r.u[1] : ur;
        r.a[3] = last ? r.a[1] : ar;
        return r;
    };
    const float wr = k.wb[0], wg = k.wb[1], wbl = k.wb[2];
    HlRow w[4];                          /* rows 2q - 1 .. 2q + 2 */
    {
        const uint32_t a = fetch(2 * q0 - 1), b = fetch(2 * q0);
        w[2] = row(a, 1);
        w[3] = row(b, 0);
    }
    uint32_t next[2] = { fetch(2 * q0 + 1), fetch(2 * q0 + 2) };
#pragma unroll 1
    for (int q = q0; q < q1; q++) {
        w[0] = w[2];
        w[1] = w[3];
        w[2] = row(next[0], 1);
        w[3] = row(next[1], 0);
        next[0] = fetch(2 * q + 3);
        next[1] = fetch(2 * q + 4);
        float out[2][2];
        out[0][0] = w[1].u[1] * wr;
        out[0][1] = w[1].u[2] * wg;
        out[1][0] = w[2].u[1] * wg;
        out[1][1] = w[2].u[2] * wbl;
        if (mine && (w[1].a[1] > 0.0f || w[1].a[2] > 0.0f || w[2].a[1] > 0.0f || w[2].a[2] > 0.0f)) {
#define U(r, c) w[r].u[c]
#define A(r, c) w[r].a[c]
            float lf[2];
            bilinear(reinterpret_cast<const float4 *>(io.levels) + k.off[0], k.lw[0], k.lh[0],
                     (float)qx * 0.5f - 0.25f, (float)q * 0.5f - 0.25f, false, lf);
            /* R at cell (1, 1): G on the cross, B on the diagonals. */
            if (A(1, 1) > 0.0f) {
                float sg = 0.0f, mg = 0.0f, sb = 0.0f, mb = 0.0f;
                sb += U(0, 0) * wbl; mb = fmax0(mb, A(0, 0));
                sg += U(0, 1) * wg;  mg = fmax0(mg, A(0, 1));
                sb += U(0, 2) * wbl; mb = fmax0(mb, A(0, 2));
                sg += U(1, 0) * wg;  mg = fmax0(mg, A(1, 0));
                sg += U(1, 2) * wg;  mg = fmax0(mg, A(1, 2));
                sb += U(2, 0) * wbl; mb = fmax0(mb, A(2, 0));
                sg += U(2, 1) * wg;  mg = fmax0(mg, A(2, 1));
                sb += U(2, 2) * wbl; mb = fmax0(mb, A(2, 2));
                out[0][0] = lift(out[0][0], A(1, 1), sg, 0.25f, mg, sb, 0.25f, mb, 0.0f, lf[1], lf[0]);
            }
            /* Gr at cell (1, 2): R left and right, B above and below. */
            if (A(1, 2) > 0.0f) {
                float sr = 0.0f, mr = 0.0f, sb = 0.0f, mb = 0.0f;
                sb += U(0, 2) * wbl; mb = fmax0(mb, A(0, 2));
                sr += U(1, 1) * wr;  mr = fmax0(mr, A(1, 1));
                sr += U(1, 3) * wr;  mr = fmax0(mr, A(1, 3));
                sb += U(2, 2) * wbl; mb = fmax0(mb, A(2, 2));
                out[0][1] = lift(out[0][1], A(1, 2), sr, 0.5f, mr, sb, 0.5f, mb, lf[0], lf[1], 0.0f);
            }
            /* Gb at cell (2, 1): R above and below, B left and right. */
            if (A(2, 1) > 0.0f) {
                float sr = 0.0f, mr = 0.0f, sb = 0.0f, mb = 0.0f;
                sr += U(1, 1) * wr;  mr = fmax0(mr, A(1, 1));
                sb += U(2, 0) * wbl; mb = fmax0(mb, A(2, 0));
                sb += U(2, 2) * wbl; mb = fmax0(mb, A(2, 2));
                sr += U(3, 1) * wr;  mr = fmax0(mr, A(3, 1));
                out[1][0] = lift(out[1][0], A(2, 1), sr, 0.5f, mr, sb, 0.5f, mb, lf[0], lf[1], 0.0f);
            }
            /* B at cell (2, 2): R on the diagonals, G on the cross. */
            if (A(2, 2) > 0.0f) {
                float sr = 0.0f, mr = 0.0f, sg = 0.0f, mg = 0.0f;
                sr += U(1, 1) * wr;  mr = fmax0(mr, A(1, 1));
                sg += U(1, 2) * wg;  mg = fmax0(mg, A(1, 2));
                sr += U(1, 3) * wr;  mr = fmax0(mr, A(1, 3));
                sg += U(2, 1) * wg;  mg = fmax0(mg, A(2, 1));
                sg += U(2, 3) * wg;  mg = fmax0(mg, A(2, 3));
                sr += U(3, 1) * wr;  mr = fmax0(mr, A(3, 1));
                sg += U(3, 2) * wg;  mg = fmax0(mg, A(3, 2));
                sr += U(3, 3) * wr;  mr = fmax0(mr, A(3, 3));
                out[1][1] = lift(out[1][1], A(2, 2), sr, 0.25f, mr, sg, 0.25f, mg, lf[0], 0.0f, lf[1]);
            }
#undef U
#undef A
        }
        __syncwarp();
        if (mine)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const __half2 hv = __floats2half2_rn(out[r][0], out[r][1]);
                if (craw_in_bounds(x0 >= 0 && x0 + 1 < k.width && 2 * q + r < k.height, io.err))
                    *reinterpret_cast<__half2 *>((char *)io.dst + (size_t)(2 * q + r) * io.dst_pitch +
                                                 (size_t)x0 * 2) = hv;
            }
    }
}

/* The rows of k_hl_fill's segments: the fewest of 2, 4 and 8 that are at most
 * kFillWaves waves of warps. A frame's highlights and bilinear develop with 8,
 * 4 and 2: 320x240 33, 29 and 27 us; 1280x720 45, 40 and 40; 2560x1440 73, 69
 * and 69; 3840x2160 121, 119 and 121. */
int fill_rows(int nx, int qh)
{
    int seg = 2;
    while (seg < kFillMost && (int64_t)nx * ((qh + seg - 1) / seg) > 152 * kFillCtas * kWalkWarps * kFillWaves)
        seg *= 2;
    return seg;
}

/* Segments of one wave of `ctas` CTAs an SM for strips of `cols` quads, a
 * multiple of 2 quad rows (texels have two), at least 4 (6 rows more are read
 * for each: 320x240 with 8 37 us, with 4 33, 1600x900 with 2 52 and with 4 50);
 * returns the CTAs. */
int hl_grid(HlGrid &g, int qw, int qh, int cols, int ctas)
{
    g.nx = (qw + cols - 1) / cols;
    const int room = 152 * ctas * kWalkWarps / g.nx, n = room > 1 ? room : 1;
    g.seg = ((qh + n - 1) / n + 1) / 2 * 2;
    g.seg = g.seg < 4 ? 4 : g.seg;
    return (g.nx * ((qh + g.seg - 1) / g.seg) + kWalkWarps - 1) / kWalkWarps;
}

dim3 grid2(int w, int h) { return dim3((w + 31) / 32, (h + 7) / 8); }

} // namespace

extern "C" int64_t craw_k_highlight_levels(int32_t width, int32_t height, CRAWKHighlight *k)
{
    int64_t total = 0;
    int n = 0;
    for (int lw = (width + 3) / 4, lh = (height + 3) / 4;; lw = (lw + 1) / 2, lh = (lh + 1) / 2) {
        if (n == CRAW_K_HL_LEVELS)
            return -1;
        k->lw[n] = lw;
        k->lh[n] = lh;
        k->off[n] = total;
        total += (int64_t)lw * lh;
        n++;
        if (lw == 1 && lh == 1)
            break;
    }
    k->nb_levels = n;
    return total;
}

extern "C" int craw_k_highlights(const CRAWKHighlight *k, const CRAWKHighlightIO *io, cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    const int qw = k->width / 2, qh = k->height / 2;
    const dim3 blk(32, 8);
    HlGrid g;
    int ctas = hl_grid(g, qw, qh, 2 * kL0N, kL0Ctas);
    k_hl_level0<<<ctas, kWalkNT, 0, s>>>(*k, *io, g);
    /* The levels from lc up are small enough for one CTA. */
    int lc = 0;
    while (lc + 1 < k->nb_levels && (int64_t)k->lw[lc] * k->lh[lc] > kCoarseTexels)
        lc++;
    if (cudaGetLastError() != cudaSuccess)
        return -5;
    /* Each launch is ready when the one before it ends (a 6000x4000 frame
     * with its develop: 429 us, 448 with plain launches). */
    for (int l = 0; l < lc; l++)
        if (craw_launch_early(k_hl_pull, grid2(k->lw[l + 1], k->lh[l + 1]), blk, 0, true, s, *k, *io, l) < 0)
            return -5;
    if (k->nb_levels > 1 && craw_launch_early(k_hl_coarse, 1, kCoarseThreads, 0, true, s, *k, *io, lc) < 0)
        return -5;
    for (int l = lc - 1; l >= 0; l--)
        if (craw_launch_early(k_hl_push, grid2(k->lw[l], k->lh[l]), blk, 0, true, s, *k, *io, l) < 0)
            return -5;
    g.nx = (qw + kFillN - 1) / kFillN;
    g.seg = fill_rows(g.nx, qh);
    ctas = (g.nx * ((qh + g.seg - 1) / g.seg) + kWalkWarps - 1) / kWalkWarps;
    return craw_launch_early(k_hl_fill, ctas, kWalkNT, 0, true, s, *k, *io, g);
}
