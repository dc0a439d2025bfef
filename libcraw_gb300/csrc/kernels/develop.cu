/*
 * The fused develop kernels (walking warps in develop_walk.cuh, tile bodies
 * in develop_tile.cuh): prep + debayer + colour + AWB statistic in one launch,
 * the RCD's interior and its border in one each; and their launcher.
 */
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "develop_tile.cuh"
#include "develop_walk.cuh"
#include "tma.cuh"

/* Whether the RCD interior tiles load their mosaic by TMA (1, the
 * default) or by plain loads (0, for comparison and tests); whether the
 * frame runs by 64x16 tiles with a per-pixel border (0, for comparison and
 * tests) or by walking warps (1, the default; 2). */
extern "C" {
int craw_k_rcd_tma = 1;
int craw_k_rcd_strips = 1;
}

namespace {

using namespace craw_dev;

/* How a frame's RCD splits into QTW x QTH quad tiles: the interior ones
 * (rows r_lo..r_hi, columns c_lo..c_hi, all aprons inside the frame) go to
 * the quad kernel, the ring of the others to the per-pixel kernel, each as
 * a grid of only its own tiles. */
struct QuadGrid {
    int qx, qy;                      /* quad tiles across, down */
    int r_lo, r_hi, c_lo, c_hi;      /* the interior (empty when hi < lo) */
    int rows_full, cols_border, mid_rows;

    void init(int w, int h)
    {
        qx = (w + QTW - 1) / QTW;
        qy = (h + QTH - 1) / QTH;
        /* quad_interior(): x0 >= 6, x0 + QTW + 6 <= w, and the same in y. */
        c_lo = 1;
        c_hi = w >= QTW + 6 ? (w - QTW - 6) / QTW : -1;
        r_lo = 1;
        r_hi = h >= QTH + 6 ? (h - QTH - 6) / QTH : -1;
        const bool has_r = r_hi >= r_lo, has_c = c_hi >= c_lo;
        rows_full = has_r ? r_lo + (qy - 1 - r_hi) : qy;   /* rows with no interior tile */
        mid_rows = has_r ? r_hi - r_lo + 1 : 0;
        cols_border = has_c ? c_lo + (qx - 1 - c_hi) : qx;  /* border tiles of the other rows */
    }
    int interior_x() const { return c_hi >= c_lo ? c_hi - c_lo + 1 : 0; }
    int interior_y() const { return r_hi >= r_lo ? r_hi - r_lo + 1 : 0; }
    int border_quads() const { return rows_full * qx + mid_rows * cols_border; }

    /* Quad tile (col, row) of border tile t. */
    CRAW_DEV void border(int t, int &col, int &row) const
    {
        const bool has_r = r_hi >= r_lo, has_c = c_hi >= c_lo;
        if (t < rows_full * qx) {
            const int rr = t / qx;
            col = t % qx;
            row = (!has_r || rr < r_lo) ? rr : r_hi + 1 + (rr - r_lo);
        } else {
            t -= rows_full * qx;
            const int rr = t / cols_border, cc = t % cols_border;
            row = r_lo + rr;
            col = (!has_c || cc < c_lo) ? cc : c_hi + 1 + (cc - c_lo);
        }
    }
};

/* An interior kernel lets the border launch that follows it on the stream
 * begin at once (programmatic dependent launch): the two write disjoint
 * tiles, and the border CTAs take the SM slots that the interior leaves
 * free. The border ends no earlier than the interior, so that what comes
 * after it on the stream, or depends on it in a graph, waits for both. The
 * border and the linear kernels let the AWB histogram's publication, which
 * waits for them, be launched meanwhile. */

__global__ void __launch_bounds__(QNT)
k_develop_rcd_quads(const CRAWKDevelop k, const CRAWKDevelopIO io, const QuadGrid g)
{
    extern __shared__ __align__(16) float smem[];
    craw_let_next_start();
    rcd_quad_tile(k, io, (g.c_lo + blockIdx.x) * QTW, (g.r_lo + blockIdx.y) * QTH, smem);
}

/* ---- the same with the tile's mosaic brought in by one TMA tile copy */

/* The box: frame columns x0 - 8 .. x0 + QTW + 8 (the apron needs x0 - 6
 * .. x0 + QTW + 6; a TMA copy starts on a 16-byte boundary, and x0 - 8 is
 * a multiple of 8 samples), rows y0 - 6 .. y0 + QTH + 6. Interior tiles
 * only, so every coordinate is inside the frame except, at most, the last
 * two columns (read as zeros and never used). */
constexpr int kBoxW = QTW + 16, kBoxH = QTH + 12;
constexpr uint32_t kBoxBytes = kBoxW * kBoxH * 2;

__global__ void __launch_bounds__(QNT)
k_develop_rcd_quads_tma(const CRAWKDevelop k, const CRAWKDevelopIO io, const QuadGrid g,
                        const __grid_constant__ CUtensorMap tmap)
{
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(8) uint64_t bar_s;
    craw_let_next_start();
    const int x0 = (g.c_lo + blockIdx.x) * QTW, y0 = (g.r_lo + blockIdx.y) * QTH;
    RcdQuads<QTW, QTH, QNT> t;
    t.carve(smem);
    /* The box lives in the discrimination planes' space, which the tile
     * first writes after the load; 128-byte aligned for the copy. */
    static_assert(kBoxBytes + 128 <= 4 * RcdQuads<QTW, QTH, QNT>::DN * sizeof(float), "box fits");
    uint32_t *box = reinterpret_cast<uint32_t *>(((uintptr_t)t.Dp + 127) & ~(uintptr_t)127);
    craw_tma::bar_init(&bar_s);
    if (threadIdx.x == 0)
        craw_tma::load_2d(box, &tmap, x0 - 8, y0 - 6, &bar_s, kBoxBytes);
    if (!__syncthreads_and(craw_tma::wait(&bar_s, 0))) {
        /* Never expected: record it, give the copy one more bound to land
         * before the CTA leaves, and skip the tile. */
        if (threadIdx.x == 0 && io.err)
            atomicOr(io.err, CRAW_K_ERR_TMA_WAIT);
        (void)craw_tma::wait(&bar_s, 0);
        return;
    }
    t.load_box<kBoxW>(k, io, box);
    __syncthreads();
    t.run();
    epilogue<QTW, QTH, QNT>(k, io, x0, y0, t.rgb);
}

/* The interior by walking warps (develop_walk.cuh), WALK_CTAS CTAs an SM:
 * 168 registers a thread and no spills (four CTAs an SM: 128 registers, up
 * to 340 bytes of spills). */
constexpr int WALK_CTAS = 3;

template <int FMT, int RGC, bool MORE>
__global__ void __launch_bounds__(WALK_NT, WALK_CTAS)
k_develop_rcd_walk(const CRAWKDevelop k, const CRAWKDevelopIO io, const WalkGrid g)
{
    __shared__ WalkSmem<RW_NQ> smem[WALK_WARPS];
    craw_await_previous();
    craw_let_next_start();
    const int warp = threadIdx.x >> 5;
    rcd_walk<FMT, RGC, MORE>(k, io, g, blockIdx.x * WALK_WARPS + warp, smem[warp]);
}

/* The border's parts and the first warp of each. */
struct RingGrid {
    WalkGrid g[4];
    int first[5];
};

/* The border by walking warps, in the same CTAs. */
template <int FMT, int RGC, bool MORE>
__global__ void __launch_bounds__(WALK_NT, WALK_CTAS)
k_develop_rcd_ring(const CRAWKDevelop k, const CRAWKDevelopIO io, const __grid_constant__ RingGrid ring)
{
    __shared__ WalkSmem<RW_NQ> smem[WALK_WARPS];
    if (io.awb.hist)
        craw_let_next_start();
    const int warp = threadIdx.x >> 5;
    const int wid = blockIdx.x * WALK_WARPS + warp;
    int part = 0;
#pragma unroll
    for (int i = 1; i < 4; i++)
        if (wid >= ring.first[i])
            part = i;
    if (wid < ring.first[4])
        ring_walk<FMT, RGC, MORE>(k, io, ring.g[part], wid - ring.first[part], smem[warp]);
    craw_await_previous();
}

/* The per-pixel RCD on the ring of border quad tiles, BTW x BTH pixels a
 * CTA (QTW / BTW of them a quad tile). */
__global__ void __launch_bounds__(256, 8)
k_develop_rcd_border(const CRAWKDevelop k, const CRAWKDevelopIO io, const QuadGrid g)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int PER = QTW / BTW;
    static_assert(QTH == BTH, "a border quad tile is one row of per-pixel tiles");
    int col, row;
    g.border(blockIdx.x / PER, col, row);
    const int x0 = col * QTW + (blockIdx.x % PER) * BTW, y0 = row * QTH;
    if (x0 < k.width)
        pixel_tile<kRcd, BTW, BTH, 256>(k, io, x0, y0, smem);
    craw_await_previous();
}

/* Every bilinear and MHC frame: CTAs an SM (5 of 96 registers for MHC and 6
 * of 80 for bilinear, a few spilled, run 7 % faster at 5760x3240 than 4 and
 * 5 without a spill). */
template <int METHOD, int EPI> constexpr int linear_ctas()
{
    return EPI == LW_ANY ? 3 : (METHOD == kMhc ? 5 : 6);
}

template <int METHOD, int EPI>
__global__ void __launch_bounds__(WALK_NT, (linear_ctas<METHOD, EPI>()))
k_develop_walk(const CRAWKDevelop k, const CRAWKDevelopIO io, const WalkGrid g)
{
    craw_await_previous();
    if (io.awb.hist)
        craw_let_next_start();
    LinearWalk<METHOD, EPI> t(k, io);
    t.run(g, blockIdx.x * WALK_WARPS + (threadIdx.x >> 5));
}

/* The RCD of a w x h frame as strips: the interior's (w, its CTAs in inner;
 * none if the frame has none) and the border's. Segments are a multiple of
 * `unit` quad rows. Either the interior takes one wave of WALK_CTAS
 * CTAs an SM and the border, in segments as short as one wave of it allows,
 * the next; or both share a wave, the border in segments half as long as the
 * interior's (its steps take longer). A segment of n rows takes n + 6 steps,
 * n + 5 in the border: the fewer in all. Frame times, sharing against taking
 * turns: 115 and 124 us (1920x1080, denoise with history, AP0), 280 and 284
 * (4098x2162, denoise); 737 and 706 (5760x3240, exact denoise, AP1). */
void rcd_grids(int width, int height, int unit, WalkGrid &w, RingGrid &ring, int &inner, int &border)
{
    const int h2 = height / 2, room = craw_sm_count() * WALK_CTAS;
    w = rcd_part(width, height, 0);
    for (int i = 0; i < 4; i++)
        ring.g[i] = rcd_part(width, height, 1 + i);
    const bool in = w.nqx > 0 && w.nqy > 0;
    auto ctas = [](int warps) { return (warps + WALK_WARPS - 1) / WALK_WARPS; };
    auto cut_ring = [&](int most) {
        ring.first[0] = 0;
        for (int i = 0; i < 4; i++)
            ring.first[i + 1] = ring.first[i] + walk_cut(ring.g[i], most, unit);
        return ctas(ring.first[4]);
    };
    auto more = [&](int n) { return n < 4 ? 4 : n + 4; };
    auto half = [&](int n) { return n / 8 * 4 > unit ? n / 8 * 4 : unit; };
    int turn = unit, turn_ring = unit, both = unit;
    while (turn < h2 && ctas(walk_cut(w, turn, unit)) > room)
        turn = more(turn);
    while (turn_ring < h2 && cut_ring(turn_ring) > room)
        turn_ring = more(turn_ring);
    while (both < h2 && ctas(walk_cut(w, both, unit)) + cut_ring(half(both)) > room)
        both = more(both);
    const bool share = in && both + 6 < turn + 6 + turn_ring + 5;
    inner = ctas(walk_cut(w, share ? both : turn, unit));
    border = cut_ring(share ? half(both) : turn_ring);
}

template <int METHOD, int EPI>
int launch_linear(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    WalkGrid g;
    g.qx0 = g.qy0 = 0;
    g.nqx = k->width / 2;
    g.nqy = k->height / 2;
    g.nx = (k->width + LW_P * LW_N - 1) / (LW_P * LW_N);
    const unsigned grid = walk_segments(g, craw_sm_count(), linear_ctas<METHOD, EPI>(), walk_unit(*io, 1));
    return craw_launch_early(k_develop_walk<METHOD, EPI>, (int)grid, WALK_NT, 0, early, s, *k, *io, g);
}

template <int METHOD>
int launch_linear(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    if (io->quarter && io->inter)
        return launch_linear<METHOD, LW_CHROMA>(k, io, early, s);
    if (io->inter || !io->dst)
        return launch_linear<METHOD, LW_ANY>(k, io, early, s);
    switch (io->dst_fmt) {
    case CRAW_K_OUT_RGBA16F: return launch_linear<METHOD, CRAW_K_OUT_RGBA16F>(k, io, early, s);
    case CRAW_K_OUT_RGB32F:  return launch_linear<METHOD, CRAW_K_OUT_RGB32F>(k, io, early, s);
    default:                 return launch_linear<METHOD, CRAW_K_OUT_RGBA32F>(k, io, early, s);
    }
}

/* The RCD kernels' shared-memory sizes, set once per device; this also
 * loads them, so that a pipeline's first frame does not wait for it. */
int prepare_rcd()
{
    constexpr size_t smem = RcdQuads<QTW, QTH, QNT>::floats * sizeof(float);
    static std::atomic<uint64_t> attr_plain{ 0 }, attr_tma{ 0 };
    if (craw_smem_attr(k_develop_rcd_quads, smem, attr_plain) < 0 ||
        craw_smem_attr(k_develop_rcd_quads_tma, smem, attr_tma) < 0)
        return -5;
    return 0;
}

/* The walking kernels of a frame. */
template <int FMT, int RGC, bool MORE>
int launch_walk(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    WalkGrid w;
    RingGrid ring;
    int inner, border;
    rcd_grids(k->width, k->height, walk_unit(*io, 2), w, ring, inner, border);
    if (inner > 0) {
        if (craw_launch_early(k_develop_rcd_walk<FMT, RGC, MORE>, inner, WALK_NT, 0, early, s, *k, *io, w) < 0)
            return -5;
    }
    return craw_launch_early(k_develop_rcd_ring<FMT, RGC, MORE>, border, WALK_NT, 0, inner > 0, s, *k, *io, ring);
}

template <int RGC>
int launch_walk(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    switch (io->dst_fmt) {
    case CRAW_K_OUT_RGBA16F: return launch_walk<CRAW_K_OUT_RGBA16F, RGC, false>(k, io, early, s);
    case CRAW_K_OUT_RGB32F:  return launch_walk<CRAW_K_OUT_RGB32F, RGC, false>(k, io, early, s);
    default:                 return launch_walk<CRAW_K_OUT_RGBA32F, RGC, false>(k, io, early, s);
    }
}

int launch_rcd(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    constexpr size_t smem = RcdQuads<QTW, QTH, QNT>::floats * sizeof(float);
    if (prepare_rcd() < 0)
        return -5;
    if (craw_k_rcd_strips) {
        if (k->fp16 || io->inter || io->quarter || !io->dst)
            return launch_walk<0, -1, true>(k, io, early, s);
        return k->color.flags & CRAW_K_COLOR_RGC ? launch_walk<1>(k, io, early, s) : launch_walk<0>(k, io, early, s);
    }
    QuadGrid g;
    g.init(k->width, k->height);
    const bool interior = g.interior_x() > 0 && g.interior_y() > 0;
    if (interior) {
        const dim3 grid(g.interior_x(), g.interior_y());
        CUtensorMap tmap;
        if (craw_k_rcd_tma && craw_tmap_u16(io->src, io->src_pitch, k->width, k->height, kBoxW, kBoxH, &tmap))
            k_develop_rcd_quads_tma<<<grid, QNT, smem, s>>>(*k, *io, g, tmap);
        else
            k_develop_rcd_quads<<<grid, QNT, smem, s>>>(*k, *io, g);
        if (cudaGetLastError() != cudaSuccess)
            return -5;
    }
    return g.border_quads() > 0 ? craw_launch_early(k_develop_rcd_border, g.border_quads() * (QTW / BTW), 256,
                                                PixelSmem<kRcd, BTW, BTH, 256>::floats * sizeof(float), interior, s,
                                                *k, *io, g)
                                : 0;
}

} // namespace

extern "C" int craw_k_develop_prepare(int method)
{
    (void)craw_sm_count();
    if (method == kRcd)
        return prepare_rcd();
    return 0;
}

extern "C" int craw_k_develop(const CRAWKDevelop *k, const CRAWKDevelopIO *io, int early,
                              cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    switch (k->method) {
    case kBilinear: return launch_linear<kBilinear>(k, io, early, s);
    case kMhc:      return launch_linear<kMhc>(k, io, early, s);
    case kRcd:      return launch_rcd(k, io, early, s);
    default:        return -22;
    }
}
