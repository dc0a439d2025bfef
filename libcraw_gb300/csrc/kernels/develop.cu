/*
 * The fused develop stage's launcher, and its RCD by walking warps
 * (develop_walk.cuh): prep + debayer + colour + AWB statistic, the interior and
 * the border in one launch each. The bilinear and MHC frames are
 * develop_linear.cu's, the small RCD frames by tiles develop_rcd_tiles.cu's.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "develop_parts.h"
#include "develop_walk.cuh"

/* Whether the RCD interior tiles load their mosaic by TMA (1, the
 * default) or by plain loads (0, for comparison and tests); whether the
 * frame runs by 64x16 tiles with a per-pixel border (0) or by walking warps
 * (2), for comparison and tests, or as rcd_by_tiles() says (1, the default). */
extern "C" {
int craw_k_rcd_tma = 1;
int craw_k_rcd_strips = 1;
}

namespace {

using namespace craw_dev;

/* An interior kernel lets the border launch that follows it on the stream
 * begin at once (programmatic dependent launch): the two write disjoint
 * tiles, and the border CTAs take the SM slots that the interior leaves
 * free. The border ends no earlier than the interior, so that what comes
 * after it on the stream, or depends on it in a graph, waits for both. The
 * border and the linear kernels let the AWB histogram's publication, which
 * waits for them, be launched meanwhile. */

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

/* Frames that tiles develop sooner than walking warps (the same bits). The
 * gamut compression lengthens a warp's steps, and where a frame has work for
 * a wave or less, its time is a segment's chain of steps; a tile has a thread
 * a quad. RGBA32F, no denoise before it (after one the walk starts early, the
 * tiles do not); us by tiles and by walking warps:
 *                                  512x288    640x362    960x540   1280x720
 *   AP1                            11.8 11.0  11.5 12.5  14.5 16.5  22.2 20.8
 *   AP1, FP16 storage              12.3 12.4  11.7 14.5  14.5 18.6  22.1 24.9
 *   AP1, AWB                       14.7 16.4  15.0 18.6  18.6 20.8  28.1 27.2
 *   BT.709                         10.5 10.3  10.6 12.4  14.5 12.6  18.7 16.5
 * (1920x1080: 37.2 31.9, 37.7 39.1, 43.3 40.6, 35.2 23.7.) Not where the
 * border is two tiles wide (1026x578, AP1: 20.6 18.5), nor for the chroma
 * path. */
constexpr int64_t kTilesLeast = 180000, kTilesMost = 800000, kTilesMostMore = 1000000;

bool rcd_by_tiles(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool more, bool early)
{
    const int64_t px = (int64_t)k->width * k->height;
    auto one_wide = [](int n, int tile) { return n % tile == 0 || n % tile >= 6; };
    return (k->color.flags & CRAW_K_COLOR_RGC) && !io->quarter && !early &&
           px <= (more ? kTilesMostMore : kTilesMost) && (px >= kTilesLeast || io->awb.hist) &&
           one_wide(k->width, QTW) && one_wide(k->height, QTH);
}

int launch_rcd(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    const bool more = k->fp16 || io->inter || io->quarter || !io->dst;
    if (craw_k_rcd_strips == 0 || (craw_k_rcd_strips == 1 && rcd_by_tiles(k, io, more, early)))
        return craw_develop_rcd_tiles(k, io, s);
    if (more)
        return launch_walk<0, -1, true>(k, io, early, s);
    return k->color.flags & CRAW_K_COLOR_RGC ? launch_walk<1>(k, io, early, s) : launch_walk<0>(k, io, early, s);
}

} // namespace

/* A debayer's kernels are a module each, which the runtime loads whole where
 * the first of them is asked for: some hundred microseconds, here rather
 * than in a pipeline's first frame. */
extern "C" int craw_k_develop_prepare(int method, int32_t width, int32_t height)
{
    cudaFuncAttributes a;
    (void)craw_sm_count();
    if (method != kRcd)
        return craw_develop_linear_prepare();
    /* Whatever the pipeline's own output space: a frame may ask for another. */
    if ((int64_t)width * height <= kTilesMostMore && craw_develop_rcd_tiles_prepare() < 0)
        return -5;
    return cudaFuncGetAttributes(&a, k_develop_rcd_walk<CRAW_K_OUT_RGBA32F, 0, false>) == cudaSuccess ? 0 : -5;
}

extern "C" int craw_k_develop(const CRAWKDevelop *k, const CRAWKDevelopIO *io, int early,
                              cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    switch (k->method) {
    case kBilinear:
    case kMhc:      return craw_develop_linear(k, io, early, s);
    case kRcd:      return launch_rcd(k, io, early, s);
    default:        return -22;
    }
}
