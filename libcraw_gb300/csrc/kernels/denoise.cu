/*
 * The raw-domain denoise kernel: one CTA per tile of the four CFA planes
 * (the tile body is denoise_tile.cuh), and its launcher.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "denoise_history.cuh"

/* Whether the packed spatial kernels bring interior tiles in by TMA (1,
 * the default) or by plain loads (0, for comparison and tests). */
extern "C" {
int craw_k_dn_tma = 1;
}

namespace {

using namespace craw_dn;

/* Four CTAs an SM where the search runs by rows (SearchRows). MARK: the
 * exact rounding's marks (spatial denoise only). TMA: interior
 * tiles bring their mosaic in by one TMA tile copy (`tmap`; spatial
 * filtering without a temporal state only). */
template <int BW, int M, int WP, bool SPATIAL, bool TEMPORAL, bool HISTORY, bool X2, bool MARK, bool TMA>
__global__ void __launch_bounds__(Cfg<BW, M, WP, SPATIAL, TEMPORAL, HISTORY>::NT, X2 && M == 8 && !HISTORY && !MARK ? 4 : 0)
k_denoise(const CRAWKDenoise k, const CRAWKDenoiseIO io, const CRAWKRound rd,
          const __grid_constant__ CUtensorMap tmap, uint32_t *err)
{
    extern __shared__ __align__(16) float smem[];
    /* Not before the rounding kernels, whose first CTAs have the work: early
     * ones gather on the SMs that are free first (720 against 708 us a frame
     * of 5760x3240). */
    if (!MARK)
        craw_let_next_start();
    denoise_tile<BW, M, WP, SPATIAL, TEMPORAL, HISTORY, X2, true, MARK, TMA>(k, io, blockIdx.x, blockIdx.y, smem,
                                                                           &rd, &tmap, err);
}

template <int BW, int M, int WP, bool SPATIAL, bool TEMPORAL, bool HISTORY, bool X2, bool MARK, bool TMA>
int go(const CRAWKDenoise *k, const CRAWKDenoiseIO *io, const CRAWKRound *rd, const CUtensorMap &tmap,
       uint32_t *err, cudaStream_t s)
{
    using C = Cfg<BW, M, WP, SPATIAL, TEMPORAL, HISTORY, X2, true, TMA>;
    auto fn = k_denoise<BW, M, WP, SPATIAL, TEMPORAL, HISTORY, X2, MARK, TMA>;
    const size_t smem = (size_t)C::smem_floats * sizeof(float);
    static std::atomic<uint64_t> attr_done{ 0 };
    if (craw_smem_attr(fn, smem, attr_done) < 0)
        return -5;
    dim3 grid((k->pw + C::OX - 1) / C::OX, (k->ph + C::OY - 1) / C::OY);
    const CRAWKRound none = { nullptr, nullptr, 0.0f, 0.0f };
    fn<<<grid, C::NT, smem, s>>>(*k, *io, rd ? *rd : none, tmap, err);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

/* The packed spatial kernels take the TMA fill when it is on and the
 * mosaic's layout allows a tensor map. */
template <int BW, int M, int WP, bool SPATIAL, bool TEMPORAL, bool HISTORY, bool X2, bool MARK = false>
int launch(const CRAWKDenoise *k, const CRAWKDenoiseIO *io, const CRAWKRound *rd, uint32_t *err, cudaStream_t s)
{
    if constexpr (SPATIAL && !TEMPORAL && X2) {
        using C = Cfg<BW, M, WP, SPATIAL, TEMPORAL, HISTORY, X2, true, true>;
        CUtensorMap tm;
        if (craw_k_dn_tma && craw_tmap_u16(io->src, io->src_pitch, 2 * k->pw, 2 * k->ph, C::BOX_W, C::BOX_H, &tm))
            return go<BW, M, WP, SPATIAL, TEMPORAL, HISTORY, X2, MARK, true>(k, io, rd, tm, err, s);
    }
    CUtensorMap none;
    memset(&none, 0, sizeof(none));
    return go<BW, M, WP, SPATIAL, TEMPORAL, HISTORY, X2, MARK, false>(k, io, rd, none, err, s);
}

/* ------------------------------------------------- with a history, packed */

/* The 2x8 packed shape's history path (denoise_history.cuh): the average
 * once a sample, then the tiles. 5760x3240: 95 + 490 us, against 658 us of
 * the 2x4 shape's tiles that average their own aprons (1.9 times the samples,
 * at a third of their instructions). At 1920x1080 the two take 83 us alike
 * (the second launch's start against 1.7 waves of tiles), and below the 2x4
 * shape is the faster: the autotuner times both, and they give the same
 * bits. */

__global__ void __launch_bounds__(TW_NT, TW_CTAS)
k_dn_temporal(const CRAWKDenoise k, const CRAWKDenoiseIO io, float *tv, const TemporalGrid g, uint32_t *err)
{
    craw_let_next_start();
    temporal_walk(k, io, tv, g, blockIdx.x * TW_WARPS + (threadIdx.x >> 5), err);
}

__global__ void __launch_bounds__(HistCfg::NT, 4)
k_dn_history(const CRAWKDenoise k, const CRAWKDenoiseIO io, const float *tv, int tma,
             const __grid_constant__ CUtensorMap tmap_t, const __grid_constant__ CUtensorMap tmap_v, uint32_t *err)
{
    extern __shared__ __align__(16) float smem[];
    craw_await_previous();
    craw_let_next_start();
    /* The tile copies land on 128-byte boundaries. */
    float *base = reinterpret_cast<float *>(((uintptr_t)smem + 127) & ~(uintptr_t)127);
    history_tile(k, io, tv, tma, &tmap_t, &tmap_v, blockIdx.x, blockIdx.y, base, err);
}

int launch_history(const CRAWKDenoise *k, const CRAWKDenoiseIO *io, float *tv, uint32_t *err, cudaStream_t s)
{
    using C = HistCfg;
    auto fn = k_dn_history;
    const size_t smem = (size_t)C::smem_floats * sizeof(float);
    static std::atomic<uint64_t> attr_done{ 0 };
    if (craw_smem_attr(fn, smem, attr_done) < 0)
        return -5;
    const HistPlanes P(k->pw, k->ph);
    /* Segments of about one wave, at least four rows. */
    TemporalGrid g;
    g.rows = k->ph + 2 * HR;
    g.nx = (k->pw + 2 * HR + 2 * TW_N - 1) / (2 * TW_N);
    const int room = 152 * TW_CTAS * TW_WARPS / (2 * g.nx), nseg = room > 1 ? room : 1;
    g.seg = (g.rows + nseg - 1) / nseg < 4 ? 4 : (g.rows + nseg - 1) / nseg;
    const int warps = 2 * g.nx * ((g.rows + g.seg - 1) / g.seg);
    k_dn_temporal<<<(warps + TW_WARPS - 1) / TW_WARPS, TW_NT, 0, s>>>(*k, *io, tv, g, err);
    if (cudaGetLastError() != cudaSuccess)
        return -5;
    CUtensorMap mt, mv;
    memset(&mt, 0, sizeof(mt));
    memset(&mv, 0, sizeof(mv));
    const bool tma = craw_k_dn_tma && craw_tmap_f32x4(tv, P.w, P.h, C::TX, C::TY, &mt) &&
                     craw_tmap_f32x4(tv + 4 * P.n, P.w, P.h, C::TX, C::TY, &mv);
    const dim3 grid((k->pw + C::OX - 1) / C::OX, (k->ph + C::OY - 1) / C::OY);
    return craw_launch_early(fn, grid, C::NT, smem, true, s, *k, *io, tv, (int)tma, mt, mv, err);
}

/* X2: the search in packed f32x2 arithmetic. */
template <int BW, int M, int WP, bool X2>
int dispatch(const CRAWKDenoise *k, const CRAWKDenoiseIO *io, const CRAWKRound *rd, float *tv, uint32_t *err,
             cudaStream_t s)
{
    const bool sp = k->mode & CRAW_K_DN_SPATIAL, te = k->mode & CRAW_K_DN_TEMPORAL;
    const bool hi = te && (k->mode & CRAW_K_DN_HISTORY);
    if (sp && !te && rd && rd->flags)
        return launch<BW, M, WP, true, false, false, X2, true>(k, io, rd, err, s);
    if (sp && !te)  return launch<BW, M, WP, true, false, false, X2>(k, io, rd, err, s);
    if (sp && !hi)  return launch<BW, M, WP, true, true, false, X2>(k, io, rd, err, s);
    if constexpr (X2 && M == 8) {
        if (sp && !tv)   /* no memory for the planes: the 2x4 shape's tiles, the same bits */
            return launch<2, 4, 2, true, true, true, true>(k, io, rd, err, s);
        if (sp)     return launch_history(k, io, tv, err, s);
    } else {
        if (sp)     return launch<BW, M, WP, true, true, true, X2>(k, io, rd, err, s);
    }
    if (te && !hi)  return launch<BW, M, WP, false, true, false, false>(k, io, rd, err, s);
    if (te)         return launch<BW, M, WP, false, true, true, false>(k, io, rd, err, s);
    return -22;
}

} // namespace

extern "C" size_t craw_k_denoise_planes(int32_t pw, int32_t ph)
{
    return 8 * HistPlanes(pw, ph).n * sizeof(float);
}

extern "C" int craw_k_denoise(const CRAWKDenoise *k, const CRAWKDenoiseIO *io, int shape,
                              const CRAWKRound *rd, float *planes, uint32_t *err, cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    switch (shape) {
    case CRAW_K_DN_SHAPE_2x8:    return dispatch<2, 8, 1, false>(k, io, rd, planes, err, s);
    case CRAW_K_DN_SHAPE_2x4:    return dispatch<2, 4, 2, false>(k, io, rd, planes, err, s);
    case CRAW_K_DN_SHAPE_2x8_X2: return dispatch<2, 8, 1, true>(k, io, rd, planes, err, s);
    case CRAW_K_DN_SHAPE_2x4_X2: return dispatch<2, 4, 2, true>(k, io, rd, planes, err, s);
    default:                  return -22;
    }
}
