/*
 * Chroma denoise on the quarter-resolution colour differences (reference
 * lib/ref/ref_chroma.c:22-158; the block means of its pass 1 are formed in
 * the develop kernel's epilogue). Pass 2 is a 9x9 joint bilateral on the
 * quarter grid; pass 3 puts the smoothed band back into every pixel and is
 * fused here with the AWB block statistic and the colour stage, so the
 * updated intermediate never goes to memory unless it is asked for.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "develop_walk.cuh"

namespace {

using namespace craw_dev;

constexpr int kR = 4;                       /* reference ref_chroma.c:15 */
constexpr float kInv2s2 = 1.0f / 8.0f;      /* 1 / (2 sigma_s^2), sigma_s = 2 */
constexpr float kRangeK = 0.35f, kChromaK = 0.35f, kRangeEps = 0.02f;

constexpr int BX = 32, BY = 8;              /* quarter texels per CTA */

__global__ void __launch_bounds__(BX * BY)
k_chroma_blur(const CRAWKChroma c, const void *q, size_t q_pitch, void *qf, size_t qf_pitch)
{
    __shared__ float4 t[(BY + 2 * kR) * (BX + 2 * kR)];
    craw_let_next_start();
    constexpr int SX = BX + 2 * kR;
    const int x0 = blockIdx.x * BX, y0 = blockIdx.y * BY;
    for (int i = threadIdx.x; i < (BY + 2 * kR) * SX; i += BX * BY) {
        int x = craw_mirror(x0 - kR + i % SX, c.qw), y = craw_mirror(y0 - kR + i / SX, c.qh);
        float v[3] = { 0.0f, 0.0f, 0.0f };
        if (craw_in_bounds(x >= 0 && x < c.qw && y >= 0 && y < c.qh, c.err))
            craw_load_rgb(q, q_pitch, x, y, c.fp16, v);
        t[i] = make_float4(v[0], v[1], v[2], 0.0f);
    }
    __syncthreads();
    const int lx = threadIdx.x % BX, ly = threadIdx.x / BX;
    const int x = x0 + lx, y = y0 + ly;
    if (x >= c.qw || y >= c.qh || !craw_in_bounds(x >= 0 && y >= 0, c.err))
        return;
    const float4 ctr = t[(ly + kR) * SX + lx + kR];
    const float level = fmaxf(ctr.z, 0.0f) + kRangeEps;
    const float inv_range = 1.0f / (kRangeK * level), inv_chroma = 1.0f / (kChromaK * level);
    float a0 = 0.0f, a1 = 0.0f, ws = 0.0f;
#pragma unroll
    for (int dy = -kR; dy <= kR; dy++) {
#pragma unroll
        for (int dx = -kR; dx <= kR; dx++) {
            float4 s = t[(ly + kR + dy) * SX + lx + kR + dx];
            float dg = (s.z - ctr.z) * inv_range;
            float d0 = (s.x - ctr.x) * inv_chroma, d1 = (s.y - ctr.y) * inv_chroma;
            /* The fast exponential: CUDA documents its error as at most
             * 2 + floor(|1.16 x|) ulp, i.e. under 1e-6 relative for the
             * weights that matter (|x| < 10, w > 4.5e-5 of the centre's
             * 1) and larger only for weights too small to move the
             * normalised weighted mean; the stage is held to 2e-4 against
             * the oracle (tests/test_gpu_parity.py, saturated rectangles
             * and zone plates, so large chroma differences). */
            float w = __expf(-(float)(dx * dx + dy * dy) * kInv2s2 - dg * dg - d0 * d0 - d1 * d1);
            a0 += w * s.x;
            a1 += w * s.y;
            ws += w;
        }
    }
    craw_store_rgba(qf, qf_pitch, x, y, c.fp16, a0 / ws, a1 / ws, ctr.z);
}

/* The band back into every pixel, by walking warps whose lanes own four pixel
 * columns, one quarter texel's: a pixel is bilinear between its texel and the
 * neighbours to its left or right and above or below, with weights in
 * eighths that its place in the 4x4 block fixes. The texels of three quarter
 * rows stay in the lane's registers, the neighbours' by shuffles (at the
 * frame's edge the lane's own); the epilogue is the bilinear and MHC
 * frames'.
 *
 * Bound: DRAM. The intermediate's rows come by asynchronous copies, kUpRows
 * of them on their way for each warp: 5760x3240 to RGBA32F, 604 MB, takes
 * 108 us (5.6 TB/s). Loaded a row ahead into registers it took 130 (too little
 * in flight at 16 warps an SM), two rows ahead with 12 warps 140, and by
 * 64x32 tiles of a pixel a thread, each loading its eight texels, 133. */
constexpr int kUpCtas = 4, kUpRows = 4, kUpRowBytes = 32 * LW_P * 16;

/* The colour differences of a texel before and after the blur. */
struct ChromaTexel {
    float d[2], b[2];
};

template <int EPI>
struct ChromaWalk : LinearWalk<kBilinear, EPI> {
    using W = LinearWalk<kBilinear, EPI>;
    const CRAWKChroma &c;
    const char *inter_in, *q, *qf;
    size_t in_pitch, q_pitch;
    char *ring;                  /* the warp's rows of the intermediate, kUpRows of kUpRowBytes */
    ChromaTexel t[3][3];         /* quarter rows r - 1 .. r + 1, columns left, own, right */

    CRAW_DEV ChromaWalk(const CRAWKDevelop &k, const CRAWKDevelopIO &io, const CRAWKChroma &c_) : W(k, io), c(c_) {}

    CRAW_DEV ChromaTexel texel(int r) const
    {
        ChromaTexel v = { { 0.0f, 0.0f }, { 0.0f, 0.0f } };
        const int x = this->x0 / LW_P, y = max(0, min(r, c.qh - 1));
        if (this->x0 >= 0 && x < c.qw && craw_in_bounds(y >= 0 && y < c.qh, c.err)) {
            float p[3];
            craw_load_rgb(q, q_pitch, x, y, c.fp16, p);
            v.d[0] = p[0];
            v.d[1] = p[1];
            craw_load_rgb(qf, q_pitch, x, y, c.fp16, p);
            v.b[0] = p[0];
            v.b[1] = p[1];
        }
        return v;
    }

    /* A quarter row's texels into window row i. */
    CRAW_DEV void put_texel(int i, const ChromaTexel &v)
    {
        const bool first = this->x0 == 0, last = this->x0 / LW_P == c.qw - 1;
        t[i][1] = v;
#pragma unroll
        for (int ch = 0; ch < 2; ch++) {
            const float dl = walk_left(v.d[ch]), dr = walk_right(v.d[ch]);
            const float bl = walk_left(v.b[ch]), br = walk_right(v.b[ch]);
            t[i][0].d[ch] = first ? v.d[ch] : dl;
            t[i][0].b[ch] = first ? v.b[ch] : bl;
            t[i][2].d[ch] = last ? v.d[ch] : dr;
            t[i][2].b[ch] = last ? v.b[ch] : br;
        }
    }

    /* Row y of the intermediate on its way into the ring: the warp's 128
     * pixels in 16-byte pieces (a pixel of floats, two of halves), zeros
     * outside the frame. A lane's pieces are 64 (or 32) bytes, their order
     * turned by the lane so that a quarter-warp's reads of one piece meet
     * every bank once. */
    CRAW_DEV void fetch(int y, int ylim) const
    {
        const int lane = threadIdx.x & 31, n = c.fp16 ? 2 : 4;     /* pieces a lane */
        char *to = ring + (y & (kUpRows - 1)) * kUpRowBytes;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (i >= n || y >= ylim)
                break;
            const int piece = i * 32 + lane, of = piece / n, x = this->x0 - LW_P * lane + piece * (LW_P / n);
            const bool ok = x >= 0 && x < c.width && craw_in_bounds(y >= 0 && y < c.height, c.err);
            const char *from = inter_in + (ok ? (size_t)y * in_pitch + (size_t)x * (c.fp16 ? 8 : 16) : 0);
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(to + 16 * (of * n + turned(piece & (n - 1), of)));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(at), "l"(from), "r"(ok ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    CRAW_DEV int turned(int piece, int lane) const
    {
        return c.fp16 ? piece ^ ((lane >> 2) & 1) : piece ^ ((lane >> 1) & 3);
    }
    /* The lane's pixels of row y, landed. */
    CRAW_DEV void landed(int y, float4 p[LW_P]) const
    {
        const int lane = threadIdx.x & 31;
        const char *at = ring + (y & (kUpRows - 1)) * kUpRowBytes;
        asm volatile("cp.async.wait_group %0;" :: "n"(kUpRows - 1) : "memory");
        __syncwarp();
        if (c.fp16) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float4 v = *reinterpret_cast<const float4 *>(at + 16 * (2 * lane + turned(i, lane)));
                p[2 * i] = make_float4(v.x, v.y, 0.0f, 0.0f);
                p[2 * i + 1] = make_float4(v.z, v.w, 0.0f, 0.0f);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                p[i] = *reinterpret_cast<const float4 *>(at + 16 * (4 * lane + turned(i, lane)));
        }
        __syncwarp();
    }

    /* Pixel (i, j) of the block: the expressions of the reference
     * (lib/ref/ref_chroma.c:110-158), every rounding explicit. */
    CRAW_DEV void pixel(int i, int j, float4 p, float o[3]) const
    {
        float px[3] = { p.x, p.y, p.z };
        if (c.fp16) {
            const uint32_t u = __float_as_uint(p.x), v = __float_as_uint(p.y);
            const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&u));
            const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&v));
            px[0] = lo.x;
            px[1] = lo.y;
            px[2] = hi.x;
        }
        const float tx = (i < 2 ? 0.625f : 0.125f) + 0.25f * (i & 1), ty = (j < 2 ? 0.625f : 0.125f) + 0.25f * (j & 1);
        const float w00 = (1.0f - tx) * (1.0f - ty), w10 = tx * (1.0f - ty), w01 = (1.0f - tx) * ty, w11 = tx * ty;
        const ChromaTexel &a = t[j >> 1][i >> 1], &b = t[j >> 1][(i >> 1) + 1];
        const ChromaTexel &e = t[(j >> 1) + 1][i >> 1], &f = t[(j >> 1) + 1][(i >> 1) + 1];
        const float g = px[1];
        float d[2] = { __fsub_rn(px[0], g), __fsub_rn(px[2], g) };
#pragma unroll
        for (int ch = 0; ch < 2; ch++) {
            const float lo = __fmaf_rn(w11, f.d[ch], __fmaf_rn(w01, e.d[ch],
                                       __fmaf_rn(w00, a.d[ch], __fmul_rn(w10, b.d[ch]))));
            const float lf = __fmaf_rn(w11, f.b[ch], __fmaf_rn(w01, e.b[ch],
                                       __fmaf_rn(w00, a.b[ch], __fmul_rn(w10, b.b[ch]))));
            d[ch] = __fmaf_rn(c.strength, __fsub_rn(lf, lo), d[ch]);
        }
        o[0] = __fadd_rn(g, d[0]);
        o[1] = g;
        o[2] = __fadd_rn(g, d[1]);
    }

    CRAW_DEV void up(const WalkGrid &g, int wid)
    {
        int y0, rows;
        if (!this->place(g, wid, y0, rows))
            return;
        const int r0 = y0 / 4;
        const ChromaTexel above = texel(r0 - 1), own = texel(r0);
        ChromaTexel below = texel(r0 + 1);
#pragma unroll
        for (int i = 0; i < kUpRows; i++)
            fetch(y0 + i, y0 + rows);
        put_texel(1, above);
        put_texel(2, own);
#pragma unroll 1
        for (int y = y0; y < y0 + rows; y += 4) {
#pragma unroll
            for (int i = 0; i < 3; i++) {
                t[0][i] = t[1][i];
                t[1][i] = t[2][i];
            }
            put_texel(2, below);
            below = texel(y / 4 + 2);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (y + j >= y0 + rows)
                    break;
                float4 p[LW_P];
                landed(y + j, p);
                fetch(y + j + kUpRows, y0 + rows);
                float o[LW_P][3];
#pragma unroll
                for (int i = 0; i < LW_P; i++)
                    pixel(i, j, p[i], o[i]);
                this->row(y + j, y + j + 1 == y0 + rows, j & 1, o);
            }
        }
    }
};

template <int EPI>
__global__ void __launch_bounds__(WALK_NT, kUpCtas)
k_chroma_up_color(const CRAWKDevelop k, const CRAWKDevelopIO io, const CRAWKChroma c, const void *inter,
                  size_t inter_pitch, const void *q, const void *qf, size_t q_pitch, const WalkGrid g)
{
    __shared__ __align__(16) char ring[WALK_WARPS][kUpRows * kUpRowBytes];
    craw_await_previous();
    if (io.awb.hist)
        craw_let_next_start();
    ChromaWalk<EPI> t(k, io, c);
    t.ring = ring[threadIdx.x >> 5];
    t.inter_in = (const char *)inter;
    t.in_pitch = inter_pitch;
    t.q = (const char *)q;
    t.qf = (const char *)qf;
    t.q_pitch = q_pitch;
    t.up(g, blockIdx.x * WALK_WARPS + (threadIdx.x >> 5));
}

} // namespace

extern "C" int craw_k_chroma_blur(const CRAWKChroma *c, const void *q, size_t q_pitch,
                                  void *qf, size_t qf_pitch, cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    dim3 grid((c->qw + BX - 1) / BX, (c->qh + BY - 1) / BY);
    k_chroma_blur<<<grid, BX * BY, 0, s>>>(*c, q, q_pitch, qf, qf_pitch);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int craw_k_chroma_up_color(const CRAWKDevelop *k, const CRAWKChroma *c,
                                      const void *inter, size_t inter_pitch,
                                      const void *q, const void *qf, size_t q_pitch,
                                      void *dst, size_t dst_pitch, int dst_fmt,
                                      void *inter_out, const CRAWKAwbOut *awb, cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    CRAWKDevelopIO io;
    memset(&io, 0, sizeof(io));
    io.dst = dst;
    io.dst_pitch = dst_pitch;
    io.dst_fmt = dst_fmt;
    io.inter = inter_out;
    io.inter_pitch = inter_pitch;
    io.awb = *awb;
    io.err = c->err;
    WalkGrid g;
    g.qx0 = g.qy0 = 0;
    g.nqx = c->width / 2;
    g.nqy = c->height / 2;
    g.nx = (c->width + LW_P * LW_N - 1) / (LW_P * LW_N);
    const unsigned ctas = walk_segments(g, craw_sm_count(), kUpCtas, awb->hist ? 4 : 2);
    auto kernel = k_chroma_up_color<LW_ANY>;
    if (!inter_out)
        kernel = dst_fmt == CRAW_K_OUT_RGBA16F  ? k_chroma_up_color<CRAW_K_OUT_RGBA16F>
                 : dst_fmt == CRAW_K_OUT_RGB32F ? k_chroma_up_color<CRAW_K_OUT_RGB32F>
                                                : k_chroma_up_color<CRAW_K_OUT_RGBA32F>;
    return craw_launch_early(kernel, (int)ctas, WALK_NT, 0, true, s, *k, io, *c, inter, inter_pitch, q, qf, q_pitch,
                             g);
}
