/*
 * The bilinear and MHC frames of the develop stage, by walking warps
 * (develop_walk.cuh): prep + debayer + colour + AWB statistic, or the chroma
 * path's intermediate and block means, in one launch.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "develop_parts.h"
#include "develop_walk.cuh"

namespace {

using namespace craw_dev;

/* Every bilinear and MHC frame: CTAs an SM (5 of 96 registers for MHC and 6
 * of 80 for bilinear, a few spilled, run 7 % faster at 5760x3240 than 4 and
 * 5 without a spill). With a kept intermediate bilinear takes 121 us a
 * 5760x3240 frame with 4 (RGBA32F, no AWB) and 128 with 3, MHC of RGB32F 117
 * with 4 and 108 with 3. */
template <int METHOD, int EPI> constexpr int linear_ctas()
{
    return EPI == LW_ANY ? (METHOD == kMhc ? 3 : 4) : (METHOD == kMhc ? 5 : 6);
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

} // namespace

int craw_develop_linear(const CRAWKDevelop *k, const CRAWKDevelopIO *io, bool early, cudaStream_t s)
{
    return k->method == kMhc ? launch_linear<kMhc>(k, io, early, s) : launch_linear<kBilinear>(k, io, early, s);
}

int craw_develop_linear_prepare()
{
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, k_develop_walk<kMhc, CRAW_K_OUT_RGBA32F>) == cudaSuccess ? 0 : -5;
}
