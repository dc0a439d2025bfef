/*
 * Batched development of frames of uneven sizes in one launch a phase.
 *
 * The work is a list of items: every denoise tile of every frame, then
 * every develop item of every frame: of an RCD batch the segments that a
 * walking warp takes of a strip (develop_walk.cuh), of the interiors first
 * (the longer ones), then of the borders; of the others 64x16 tiles. Each
 * runs the same body as the single-frame kernels (denoise_tile.cuh,
 * develop_walk.cuh, develop_tile.cuh) on its frame's constants, which sit in
 * the launch's parameter bank (the frame table is a __grid_constant__
 * parameter): uniform constant-cache loads, as the single-frame kernels read
 * theirs. A CTA takes one item (four, a warp each, of an RCD batch's develop
 * phase), so that the hardware hands the next out as a CTA ends; CTAs that
 * kept to items blockIdx.x + k gridDim.x left a tenth of a preview batch's
 * denoise time to a last round that was nearly empty.
 *
 * Fused, one persistent cooperative launch does both phases: between them
 * every CTA waits at the cooperative-groups barrier (the runtime checks that
 * the whole grid is resident), because a develop item reads its neighbours'
 * denoised samples. Unfused, the phases are two launches.
 */
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "denoise_tile.cuh"
#include "develop_tile.cuh"
#include "develop_walk.cuh"

namespace {

namespace cg = cooperative_groups;
using namespace craw_dev;

constexpr int BQH = 16;     /* rows of a tile of the bilinear and MHC develop */

/* The denoise of a batch: the packed f32x2 search, 2 columns x M rows a
 * thread: the 2x8 one by 128 threads at four CTAs an SM (its search runs by
 * rows), the 2x4 one by 256. */
template <int M> struct DnShape {
    static constexpr int WP = M == 8 ? 1 : 2;
    using C = craw_dn::Cfg<2, M, WP, true, false, false, true, M == 8>;
    static constexpr int NT = C::NT, CTAS = M == 8 ? 4 : 1;
};

/* The frame an item belongs to: the last one whose first item (`first` of
 * its frame) is not after it. */
template <typename FIRST>
CRAW_DEV int item_frame(const CRAWKBatchTable &T, int nb, int item, FIRST first)
{
    int lo = 0, n = nb;
    while (n > 1) {
        const int h = n / 2;
        if (first(T.f[lo + h]) <= item) {
            lo += h;
            n -= h;
        } else {
            n = h;
        }
    }
    return lo;
}

template <int M>
CRAW_DEV void denoise_item(const CRAWKBatchTable &T, int nb, int it, float *smem)
{
    using D = DnShape<M>;
    const CRAWKBatchFrame &F = T.f[item_frame(T, nb, it, [](const CRAWKBatchFrame &f) { return f.dn_first; })];
    const int local = it - F.dn_first;
    craw_dn::denoise_tile<2, M, D::WP, true, false, false, true, M == 8>(F.dn, F.dio, local % F.dn_tx,
                                                                       local / F.dn_tx, smem);
}

/* A tile of a bilinear or MHC frame. */
template <int METHOD, int NT>
CRAW_DEV void develop_tile(const CRAWKBatchTable &T, int nb, int it, float *smem)
{
    const CRAWKBatchFrame &F = T.f[item_frame(T, nb, it, [](const CRAWKBatchFrame &f) { return f.dv_first; })];
    const int local = it - F.dv_first;
    const int x0 = (local % F.dv_tx) * QTW, y0 = (local / F.dv_tx) * BQH;
    /* Per-pixel tiles of BTW x BTH cover the QTW x BQH item. */
    for (int sx = 0; sx < QTW; sx += BTW) {
        if (x0 + sx >= F.dv.width)
            break;
        if (sx)
            __syncthreads();
        pixel_tile<METHOD, BTW, BTH, NT, BQH>(F.dv, F.vio, x0 + sx, y0, smem);
    }
}

/* A warp's segment of a strip of an RCD frame: the interiors', then, from
 * the first frame's dv_border on, the borders'. */
template <int FMT, bool MORE>
CRAW_DEV void develop_segment(const CRAWKBatchTable &T, int nb, int it, WalkSmem<RW_NQ> &smem)
{
    if (it < T.f[0].dv_border) {
        const CRAWKBatchFrame &F = T.f[item_frame(T, nb, it, [](const CRAWKBatchFrame &f) { return f.dv_first; })];
        WalkGrid g = rcd_part(F.dv.width, F.dv.height, 0);
        walk_cut(g, F.dv_cut);
        rcd_walk<FMT, -1, MORE>(F.dv, F.vio, g, it - F.dv_first, smem);
    } else {
        const CRAWKBatchFrame &F = T.f[item_frame(T, nb, it, [](const CRAWKBatchFrame &f) { return f.dv_border; })];
        int wid = it - F.dv_border;
        WalkGrid g;
#pragma unroll 1
        for (int i = 1; i <= 4; i++) {
            g = rcd_part(F.dv.width, F.dv.height, i);
            const int n = walk_cut(g, F.dv_cut_border);
            if (wid < n)
                break;
            wid -= n;
        }
        ring_walk<FMT, -1, MORE>(F.dv, F.vio, g, wid, smem);
    }
}

template <int M, int METHOD> struct Smem {
    static constexpr int NT = DnShape<M>::NT;
    static constexpr int dn = DnShape<M>::C::smem_floats;
    static constexpr int walk = NT / 32 * (int)sizeof(WalkSmem<RW_NQ>) / 4;
    static constexpr int dv = METHOD == kRcd ? walk : PixelSmem<METHOD, BTW, BTH, NT>::floats;
    static constexpr int floats = dn > dv ? dn : dv;
};

template <int M, int METHOD>
__global__ void __launch_bounds__(DnShape<M>::NT)
k_batch_fused(const __grid_constant__ CRAWKBatchTable T, int nb, int dn_items, int dv_items)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int NT = DnShape<M>::NT, WARPS = NT / 32;
    for (int it = blockIdx.x; it < dn_items; it += gridDim.x) {
        __syncthreads();   /* the previous item's shared memory is free */
        denoise_item<M>(T, nb, it, smem);
    }
    cg::this_grid().sync();
    if constexpr (METHOD == kRcd) {
        WalkSmem<RW_NQ> &mine = reinterpret_cast<WalkSmem<RW_NQ> *>(smem)[threadIdx.x >> 5];
        for (int it = blockIdx.x * WARPS + (threadIdx.x >> 5); it < dv_items; it += gridDim.x * WARPS) {
            __syncwarp();
            develop_segment<0, true>(T, nb, it, mine);
        }
    } else {
        for (int it = blockIdx.x; it < dv_items; it += gridDim.x) {
            __syncthreads();
            develop_tile<METHOD, NT>(T, nb, it, smem);
        }
    }
}

template <int M>
__global__ void __launch_bounds__(DnShape<M>::NT, DnShape<M>::CTAS)
k_batch_denoise(const __grid_constant__ CRAWKBatchTable T, int nb, int dn_items, int dv_items)
{
    extern __shared__ __align__(16) float smem[];
    denoise_item<M>(T, nb, blockIdx.x, smem);
}

constexpr int TILE_NT = 256;

template <int METHOD>
__global__ void __launch_bounds__(TILE_NT, 4)
k_batch_develop(const __grid_constant__ CRAWKBatchTable T, int nb, int dn_items, int dv_items)
{
    extern __shared__ __align__(16) float smem[];
    develop_tile<METHOD, TILE_NT>(T, nb, blockIdx.x, smem);
}

/* As the single-frame walking kernels. 48 previews of 9 Mpx in all, BT.2020
 * half float: 107 us, where 64x16 tiles in persistent CTAs (their borders a
 * pixel a thread) took 242. */
constexpr int SEG_CTAS = 3;

template <int FMT>
__global__ void __launch_bounds__(WALK_NT, SEG_CTAS)
k_batch_develop_rcd(const __grid_constant__ CRAWKBatchTable T, int nb, int dn_items, int dv_items)
{
    __shared__ WalkSmem<RW_NQ> smem[WALK_WARPS];
    const int warp = threadIdx.x >> 5, it = blockIdx.x * WALK_WARPS + warp;
    if (it < dv_items)
        develop_segment<FMT, false>(T, nb, it, smem[warp]);
}

int device_sms()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return -1;
    return sms;
}

/* As many CTAs as fit on the device at once, at most `items`. */
template <typename K>
int resident_grid(K kernel, int threads, size_t smem, int items)
{
    int per_sm = 0, sms = device_sms();
    if (sms <= 0 ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess ||
        per_sm <= 0)
        return -1;
    return items < per_sm * sms ? (items > 0 ? items : 1) : per_sm * sms;
}

template <typename K>
int set_smem(K kernel, size_t smem)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
           cudaSuccess ? 0 : -5;
}

template <typename K>
int start(K kernel, int grid, int threads, size_t smem, void **args, cudaStream_t s)
{
    if (set_smem(kernel, smem) < 0 ||
        cudaLaunchKernel((const void *)kernel, dim3(grid), dim3(threads), args, smem, s) != cudaSuccess)
        return -5;
    return 0;
}

template <int M, int METHOD>
int run(const CRAWKBatchTable *T, int nb, int dn_items, int dv_items, int fused, cudaStream_t s)
{
    void *args[] = { (void *)T, (void *)&nb, (void *)&dn_items, (void *)&dv_items };
    if (fused) {
        constexpr int NT = DnShape<M>::NT;
        const size_t smem = Smem<M, METHOD>::floats * sizeof(float);
        auto k = k_batch_fused<M, METHOD>;
        if (set_smem(k, smem) < 0)
            return -5;
        int grid = resident_grid(k, NT, smem, dn_items > dv_items ? dn_items : dv_items);
        if (grid < 0)
            return -5;
        if (cudaLaunchCooperativeKernel((const void *)k, dim3(grid), dim3(NT), args, smem, s) != cudaSuccess)
            return -5;
        return 0;
    }
    if (dn_items > 0 && start(k_batch_denoise<M>, dn_items, DnShape<M>::NT, DnShape<M>::C::smem_floats * sizeof(float),
                              args, s) < 0)
        return -5;
    if constexpr (METHOD == kRcd) {
        /* A batch's frames share their output's layout. */
        const int grid = (dv_items + WALK_WARPS - 1) / WALK_WARPS;
        switch (T->f[0].vio.dst_fmt) {
        case CRAW_K_OUT_RGBA16F: return start(k_batch_develop_rcd<CRAW_K_OUT_RGBA16F>, grid, WALK_NT, 0, args, s);
        case CRAW_K_OUT_RGB32F:  return start(k_batch_develop_rcd<CRAW_K_OUT_RGB32F>, grid, WALK_NT, 0, args, s);
        default:                 return start(k_batch_develop_rcd<CRAW_K_OUT_RGBA32F>, grid, WALK_NT, 0, args, s);
        }
    } else {
        return start(k_batch_develop<METHOD>, dv_items, TILE_NT,
                     PixelSmem<METHOD, BTW, BTH, TILE_NT>::floats * sizeof(float), args, s);
    }
}

template <int M>
int run_method(const CRAWKBatchTable *T, int nb, int dn_items, int dv_items, int method, int fused,
               cudaStream_t s)
{
    switch (method) {
    case kBilinear: return run<M, kBilinear>(T, nb, dn_items, dv_items, fused, s);
    case kMhc:      return run<M, kMhc>(T, nb, dn_items, dv_items, fused, s);
    case kRcd:      return run<M, kRcd>(T, nb, dn_items, dv_items, fused, s);
    default:        return -22;
    }
}

} // namespace

namespace {

/* An RCD batch's segments: the interiors' as short as one wave of SEG_CTAS
 * CTAs an SM allows; the borders', which follow as CTAs end, as long as the
 * steps that one of the wave's warps gets of them (a segment of n rows takes
 * n + 5). Multiples of 4 rows. */
int layout_segments(CRAWKBatchFrame *f, int nb)
{
    const int sms = device_sms(), room = (sms > 0 ? sms : 152) * SEG_CTAS * WALK_WARPS;
    WalkGrid g[CRAW_K_BATCH_MAX][5];
    long rows[2] = { 0, 0 };         /* quad rows of the strips */
    int tall = 0;
    for (int i = 0; i < nb; i++) {
        for (int p = 0; p < 5; p++) {
            g[i][p] = rcd_part(f[i].dv.width, f[i].dv.height, p);
            if (g[i][p].nqx > 0 && g[i][p].nqy > 0)
                rows[p > 0] += (long)g[i][p].nx * g[i][p].nqy;
        }
        tall = f[i].dv.height / 2 > tall ? f[i].dv.height / 2 : tall;
    }
    auto at_least = [](long n) { return n > 4 ? (int)((n + 3) / 4 * 4) : 4; };
    auto interiors = [&](int most) {
        int n = 0;
        for (int i = 0; i < nb; i++)
            n += walk_cut(g[i][0], most);
        return n;
    };
    int cut = at_least(rows[0] / room), border = 4;
    while (cut < tall && interiors(cut) > room)
        cut += 4;
    for (; border < cut; border += 4) {
        long steps = rows[1];
        for (int i = 0; i < nb; i++)
            for (int p = 1; p < 5; p++)
                steps += 5L * walk_cut(g[i][p], border);
        if (steps <= (long)(border + 5) * room)
            break;
    }
    int n = 0;
    for (int i = 0; i < nb; i++) {
        f[i].dv_cut = cut;
        f[i].dv_cut_border = border;
        f[i].dv_first = n;
        n += walk_cut(g[i][0], cut);
    }
    for (int i = 0; i < nb; i++) {
        f[i].dv_border = n;
        for (int p = 1; p < 5; p++)
            n += walk_cut(g[i][p], border);
    }
    return n;
}

} // namespace

extern "C" void craw_k_batch_layout(CRAWKBatchFrame *f, int32_t nb, int method, int32_t *dn_items, int32_t *dv_items)
{
    constexpr int ox = DnShape<8>::C::OX, oy = DnShape<8>::C::OY;
    static_assert(DnShape<4>::C::OX == ox && DnShape<4>::C::OY == oy, "both shapes' tiles alike");
    int dn = 0, dv = 0;
    for (int i = 0; i < nb; i++) {
        const int w = f[i].dv.width, h = f[i].dv.height;
        f[i].dn_tx = f[i].dn.mode ? (w / 2 + ox - 1) / ox : 0;
        f[i].dn_first = dn;
        dn += f[i].dn_tx * ((h / 2 + oy - 1) / oy);
        f[i].dv_tx = (w + QTW - 1) / QTW;
        f[i].dv_first = dv;
        dv += f[i].dv_tx * ((h + BQH - 1) / BQH);
    }
    *dn_items = dn;
    *dv_items = method == kRcd ? layout_segments(f, nb) : dv;
}

/* Both shapes filter the same tiles to the same bits. With two tiles an SM
 * or fewer 256 threads a tile end sooner (a 640x360 frame of 120 tiles, with
 * its develop: 33 us against 39); with more the 2x8 search's instructions
 * count (48 previews of 4812 tiles: 246 us against 216). */
extern "C" int craw_k_batch_shape(int32_t dn_items)
{
    const int sms = device_sms();
    return dn_items > 2 * (sms > 0 ? sms : 152) ? CRAW_K_BATCH_DN_2x8 : CRAW_K_BATCH_DN_2x4;
}

extern "C" int craw_k_batch_prepare(void)
{
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, k_batch_denoise<8>) == cudaSuccess ? 0 : -5;
}

extern "C" int craw_k_batch(const CRAWKBatchTable *table, int32_t nb, int32_t dn_items,
                            int32_t dv_items, int method, int fused, cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    if (nb <= 0 || nb > CRAW_K_BATCH_MAX)
        return -22;
    return craw_k_batch_shape(dn_items) == CRAW_K_BATCH_DN_2x8
               ? run_method<8>(table, nb, dn_items, dv_items, method, fused, s)
               : run_method<4>(table, nb, dn_items, dv_items, method, fused, s);
}

extern "C" int craw_k_batch_update(cudaGraphExec_t exec, cudaGraph_t graph, const CRAWKBatchTable *table,
                                   int32_t nb, int32_t dn_items, int32_t dv_items)
{
    cudaGraphNode_t nodes[8];
    size_t n = 8;
    void *args[] = { (void *)table, (void *)&nb, (void *)&dn_items, (void *)&dv_items };

    if (cudaGraphGetNodes(graph, nodes, &n) != cudaSuccess || n > 8)
        return -5;
    for (size_t i = 0; i < n; i++) {
        cudaGraphNodeType t;
        cudaKernelNodeParams p;
        if (cudaGraphNodeGetType(nodes[i], &t) != cudaSuccess)
            return -5;
        if (t != cudaGraphNodeTypeKernel)
            continue;
        if (cudaGraphKernelNodeGetParams(nodes[i], &p) != cudaSuccess)
            return -5;
        p.kernelParams = args;
        p.extra = nullptr;
        if (cudaGraphExecKernelNodeSetParams(exec, nodes[i], &p) != cudaSuccess)
            return -5;
    }
    return 0;
}
