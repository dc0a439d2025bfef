/*
 * The RCD by 64x16 tiles (develop_tile.cuh), where a frame is small and has the
 * gamut compression (develop.cu's rule): the interior by CFA quads, its mosaic
 * by a TMA tile copy or by plain loads, the border a pixel a thread.
 */
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "develop_parts.h"
#include "develop_tile.cuh"
#include "tma.cuh"

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

} // namespace

/* Their shared-memory sizes, set once per device, which also loads them. */
int craw_develop_rcd_tiles_prepare()
{
    constexpr size_t smem = RcdQuads<QTW, QTH, QNT>::floats * sizeof(float);
    static std::atomic<uint64_t> attr_plain{ 0 }, attr_tma{ 0 };
    return craw_smem_attr(k_develop_rcd_quads, smem, attr_plain) < 0 ||
                   craw_smem_attr(k_develop_rcd_quads_tma, smem, attr_tma) < 0
               ? -5
               : 0;
}

/* The border may begin beside the interior, and ends no earlier than it. */
int craw_develop_rcd_tiles(const CRAWKDevelop *k, const CRAWKDevelopIO *io, cudaStream_t s)
{
    constexpr size_t smem = RcdQuads<QTW, QTH, QNT>::floats * sizeof(float);
    if (craw_develop_rcd_tiles_prepare() < 0)
        return -5;
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
