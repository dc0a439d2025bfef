/*
 * Noise-model estimation, the device half (reference lib/noise.c:338-504,
 * binning 396-450; the least-trimmed-squares seed 187-250).
 *
 *   k_noise_lut     the four sites' plane values of every 16-bit code, in
 *                   double and rounded once, as the reference converts
 *   k_noise_bin     every interior position of the four planes: the 9x9
 *                   mean (81 float additions in the reference's order), its
 *                   bin, which is kept, the exact sums of the bins' means,
 *                   and a first histogram of the 3x3 |high-pass| per bin
 *                   (its top 11 bits)
 *   k_noise_select  per bin, which bucket holds the (count / 2)-th
 *                   smallest |high-pass|; two more rounds over the next
 *                   10 and last 10 bits (k_noise_refine, which forms the
 *                   high-pass again) leave its bits
 *   k_noise_lts     the trimmed cost of every pair of bins in floats, one
 *                   warp a pair, then in doubles of the pairs that the
 *                   floats leave in question; the first least one
 *
 * The median is an order statistic, so it is the reference's value
 * exactly; so are the counts. A bin's sum of means is kept as an integer
 * (each float mean times 2^64, exact for means >= 2^-40, in three 32-bit
 * words) so that it does not depend on the order the atomics land in;
 * the reference adds the same floats into a double one by one. Built
 * without multiply-add contraction, as the reference's host code is.
 */
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>

#include "common.cuh"

namespace {

constexpr int kR = 4;                                   /* radius of the plane mean */
constexpr int kB1 = 2048, kB2 = 1024, kB3 = 1024;       /* buckets: key bits 30-20, 19-10, 9-0 */
constexpr uint32_t kNone = 0xffffffffu;

/* An item of k_noise_bin: the two planes of one row parity, kCX columns by
 * kCY rows of positions; a thread has 4 columns by kNR rows of each. */
constexpr int kNR = 2, kBinWarps = 16, kBinNT = 32 * kBinWarps;
constexpr int kCX = 128, kCY = kNR * kBinWarps;
constexpr int kPW = kCX + 2 * kR, kPH = kCY + 2 * kR;   /* the staged patch of a plane */

/* The frame as the kernels see it: interior positions across and down; the
 * kept bins' row pitch; per bin, the `win` buckets from `lo` on that a CTA
 * counts in shared memory. A bin index of nb_bins means none. */
struct NoiseGrid {
    int ww, hh, wp;
    int ntx, nty;
    int win, lo;
};

NoiseGrid noise_grid(int32_t w, int32_t h, int32_t nb)
{
    NoiseGrid g;
    g.ww = w / 2 - 2 * kR;
    g.hh = h / 2 - 2 * kR;
    g.wp = (g.ww + 3) / 4 * 4;
    g.ntx = (g.ww + kCX - 1) / kCX;
    g.nty = (g.hh + kCY - 1) / kCY;
    /* The counters reach over the |high-pass| of a camera's noise, 2^-12 to
     * 2^-4 (above 256 bins 2^-10 to 2^-6): 32 KB for up to 128 bins, 64 at
     * most. The others are counted in memory. */
    g.win = nb <= 256 ? 64 : 32;
    g.lo = 8 * (nb <= 256 ? 127 - 12 : 127 - 10);
    return g;
}

size_t bin_bytes(int32_t nb)   /* a kept bin index */
{
    return nb <= 255 ? 1 : 2;
}

struct Layout {
    size_t lut, h1, h2, h3, sel, bidx, total;
};

Layout layout(int32_t w, int32_t h, int32_t nb)
{
    const NoiseGrid g = noise_grid(w, h, nb);
    Layout L;
    size_t o = 0;
    auto take = [&o](size_t bytes) {
        const size_t at = o;
        o = (o + bytes + 255) / 256 * 256;
        return at;
    };
    L.lut = take((size_t)4 * 65536 * sizeof(float));
    L.h1 = take((size_t)nb * kB1 * 4);
    L.h2 = take((size_t)nb * kB2 * 4);
    L.h3 = take((size_t)nb * kB3 * 4);
    L.sel = take((size_t)nb * 8);
    L.bidx = take((size_t)4 * g.hh * g.wp * bin_bytes(nb));
    L.total = o;
    return L;
}

/* Double arithmetic is what bounds this (two lanes of it an SM): the
 * division is one multiplication by the correctly rounded reciprocal and
 * Markstein's correction, which rounds as the division does (IBM J. Res.
 * Dev. 34(1), 1990, theorem for a correctly rounded reciprocal). */
struct NoiseSite {
    double black[4], range[4], rcp[4];
};

__global__ void __launch_bounds__(256) k_noise_lut(const __grid_constant__ NoiseSite n, float *lut)
{
    craw_let_next_start();
    const int s = blockIdx.y, raw = blockIdx.x * 256 + threadIdx.x;
    const double x = (double)raw * (1.0 / 65535.0) - n.black[s];
    const double q = x * n.rcp[s];
    lut[s * 65536 + raw] = (float)__fma_rn(__fma_rn(-n.range[s], q, x), n.rcp[s], q);
}

/* A positive float (below 2^31) times 2^64 as a 96-bit integer, in three
 * 32-bit words, truncated below 2^-64. f = m 2^(e - 150), m < 2^24. */
__device__ __forceinline__ void fixed96(float f, uint32_t w[3])
{
    const uint32_t b = __float_as_uint(f);
    const int e = (int)(b >> 23);
    const uint64_t m = (uint64_t)((b & 0x7fffffu) | 0x800000u);
    const int sh = e - 86;
    uint64_t lo = 0;
    uint32_t hi = 0;
    if (e == 0 || sh <= -24) {
    } else if (sh < 0) {
        lo = m >> -sh;
    } else if (sh <= 40) {
        lo = m << sh;
    } else if (sh < 64) {
        lo = m << sh;
        hi = (uint32_t)(m >> (64 - sh));
    } else {
        hi = (uint32_t)(m << (sh - 64));
    }
    w[0] = (uint32_t)lo;
    w[1] = (uint32_t)(lo >> 32);
    w[2] = hi;
}

/* The plane columns c .. c + 3 of mosaic row `row` as their two planes'
 * sample pairs, zeros outside the plane (w2 columns); c a multiple of 4. */
CRAW_DEV uint4 plane_quad(const char *row, int c, int w2)
{
    const uint32_t *p = reinterpret_cast<const uint32_t *>(row) + c;
    if (c >= 0 && c + 4 <= w2)
        return __ldg(reinterpret_cast<const uint4 *>(p));
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (c >= 0 && c < w2)
        v.x = __ldg(p);
    if (c >= 0 && c + 1 < w2)
        v.y = __ldg(p + 1);
    if (c >= 0 && c + 2 < w2)
        v.z = __ldg(p + 2);
    return v;
}

CRAW_DEV float4 plane_values(const float *lut, uint4 v, int sh)
{
    return make_float4(lut[(v.x >> sh) & 0xffffu], lut[(v.y >> sh) & 0xffffu], lut[(v.z >> sh) & 0xffffu],
                       lut[(v.w >> sh) & 0xffffu]);
}

/* [1 -2 1; -2 4 -2; 1 -2 1] / 6 at column c of three rows, in the
 * reference's order; its magnitude's bits. */
CRAW_DEV uint32_t high_pass(const float *n, const float *o, const float *s, int c)
{
    const float hp = (n[c - 1] + n[c + 1] + s[c - 1] + s[c + 1] -
                      2.0f * (n[c] + s[c] + o[c - 1] + o[c + 1]) + 4.0f * o[c]) * (1.0f / 6.0f);
    return __float_as_uint(fabsf(hp));
}

/* A thread's samples, in the order it visits them: neighbours mostly share
 * a bin, so their means add up in a register and reach the CTA's tallies
 * (three 17-bit words a bin) when the bin changes. */
struct BinTally {
    const CRAWKNoise &k;
    const NoiseGrid &g;
    uint32_t *hist, *tally, *h1;
    CRAWKNoiseBin *bins;
    int cur;
    uint64_t run;            /* the means' sum times 2^45 */

    CRAW_DEV void flush()
    {
        if (cur < k.nb_bins && run) {
            atomicAdd(&tally[cur], (uint32_t)run & 0x1ffffu);
            atomicAdd(&tally[k.nb_bins + cur], (uint32_t)(run >> 17) & 0x1ffffu);
            atomicAdd(&tally[2 * k.nb_bins + cur], (uint32_t)(run >> 34));
        }
    }

    /* The whole warp calls this; returns the bin. */
    CRAW_DEV int sample(float mean, uint32_t key, bool inside)
    {
        const int nb = k.nb_bins;
        int bin = nb;
        if (inside && mean > 0.0f && !(mean > k.max_level)) {
            bin = (int)(sqrtf(mean) * (float)nb);
            bin = bin < 0 ? 0 : (bin > nb - 1 ? nb - 1 : bin);
        }
        if (bin != cur) {
            flush();
            cur = bin;
            run = 0;
        }
        if (bin < nb) {
            const uint32_t b = __float_as_uint(mean);
            const int e = (int)(b >> 23);
            if (e >= 105 && e < 128) {          /* 2^-22 <= mean < 2 */
                run += (uint64_t)((b & 0x7fffffu) | 0x800000u) << (e - 105);
            } else {
                uint32_t f[3];
                fixed96(mean, f);
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (f[q])
                        atomicAdd(reinterpret_cast<unsigned long long *>(&bins[bin].sum[q]),
                                  (unsigned long long)f[q]);
            }
        }
        const uint32_t at = (key >> 20) - (uint32_t)g.lo;
        const bool in = at < (uint32_t)g.win;
        if (bin < nb && in)
            atomicAdd(&hist[bin * g.win + at], 1u);
        const unsigned out = __ballot_sync(0xffffffffu, bin < nb && !in);
        if (out) {
            /* Of many at once (a flat frame's zeros), one atomic per
             * distinct bucket. */
            const uint32_t addr = bin < nb && !in ? (uint32_t)bin * kB1 + (key >> 20) : kNone;
            const unsigned same = __popc(out) > 4 ? __match_any_sync(0xffffffffu, addr) : 1u << (threadIdx.x & 31);
            if (addr != kNone && (int)(threadIdx.x & 31) == __ffs(same) - 1)
                atomicAdd(&h1[addr], (uint32_t)__popc(same));
        }
        return bin;
    }
};

template <typename B> struct BinQuad;
template <> struct BinQuad<uint8_t> { using T = uchar4; };
template <> struct BinQuad<uint16_t> { using T = ushort4; };

/* Bound: instruction issue (the 81 additions are 40 % of the instructions),
 * near the 70 % of it that the gathers from the code table leave. A thread's
 * samples share the window they read from shared memory (7.5 16-byte loads a
 * sample), and what a sample adds to its bin stays in the thread or in shared
 * memory: 142 us at 5760x3240, where a lane a sample (81 loads, and two
 * matches and six reductions over the warp for the tallies) took 291. The
 * table wants what shared memory leaves of the L1: 4 rows a thread in three
 * CTAs of 76 KB took 217 us, in two 152; packed additions issue half as often
 * and take the adders as long: 153. */
template <typename B>
__global__ void __launch_bounds__(kBinNT, 2)
k_noise_bin(const CRAWKNoise k, const NoiseGrid g, const uint16_t *src, size_t pitch, const float *lut,
            uint32_t *h1, B *bidx, CRAWKNoiseBin *bins)
{
    extern __shared__ __align__(16) float smem[];
    float *P = smem;                                             /* [2][kPH][kPW] */
    uint32_t *hist = reinterpret_cast<uint32_t *>(smem + 2 * kPH * kPW);
    uint32_t *tally = hist + k.nb_bins * g.win;
    const int w2 = k.width / 2, h2 = k.height / 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int items = 2 * g.ntx * g.nty;

    craw_await_previous();
    craw_let_next_start();
    for (int i = tid; i < k.nb_bins * (g.win + 3); i += kBinNT)
        hist[i] = 0;                                             /* and the tallies after it */
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int py = it & 1, t = it >> 1;
        const int i0 = (t % g.ntx) * kCX, k0 = (t / g.ntx) * kCY;
        /* The patch: plane rows k0 .. k0 + kPH, columns i0 .. i0 + kPW. */
        constexpr int kVec = kPH * (kPW / 4), kIt = (kVec + kBinNT - 1) / kBinNT;
        uint4 raw[kIt];
#pragma unroll
        for (int j = 0; j < kIt; j++) {
            const int v = tid + j * kBinNT, r = v / (kPW / 4), c = 4 * (v % (kPW / 4));
            raw[j] = make_uint4(0u, 0u, 0u, 0u);
            if (v < kVec && k0 + r < h2)
                raw[j] = plane_quad((const char *)src + (size_t)(2 * (k0 + r) + py) * pitch, i0 + c, w2);
        }
        __syncthreads();                         /* the last item's patch and tallies are done with */
#pragma unroll
        for (int j = 0; j < kIt; j++) {
            const int v = tid + j * kBinNT;
            if (v < kVec)
#pragma unroll
                for (int pl = 0; pl < 2; pl++)
                    reinterpret_cast<float4 *>(P + pl * kPH * kPW)[v] =
                        plane_values(lut + (2 * py + pl) * 65536, raw[j], 16 * pl);
        }
        __syncthreads();

        const int io = i0 + 4 * lane, ko = k0 + kNR * warp;
        BinTally tl{ k, g, hist, tally, h1, bins, k.nb_bins, 0 };
#pragma unroll 1
        for (int pl = 0; pl < 2; pl++) {
            const float *p = P + pl * kPH * kPW + kNR * warp * kPW + 4 * lane;
            float acc[kNR][4], up[12], at[12];
            uint32_t key[kNR][4];
#pragma unroll
            for (int r = 0; r < kNR + 2 * kR; r++) {
                float w[12];
#pragma unroll
                for (int v = 0; v < 3; v++)
                    *reinterpret_cast<float4 *>(w + 4 * v) = reinterpret_cast<const float4 *>(p + r * kPW)[v];
                /* The mean's terms, rows then columns. */
#pragma unroll
                for (int j = 0; j < kNR; j++) {
                    if (r < j || r > j + 2 * kR)
                        continue;
#pragma unroll
                    for (int dx = 0; dx <= 2 * kR; dx++)
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            acc[j][q] = r == j && dx == 0 ? w[q] : acc[j][q] + w[q + dx];
                }
                if (r >= kR + 1 && r <= kR + kNR)
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        key[r - kR - 1][q] = high_pass(up, at, w, kR + q);
#pragma unroll
                for (int c = 0; c < 12; c++) {
                    up[c] = at[c];
                    at[c] = w[c];
                }
            }
            B *out = bidx + ((size_t)(2 * py + pl) * g.hh + ko) * g.wp + io;
#pragma unroll 1
            for (int j = 0; j < kNR; j++) {
                int b[4];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    b[q] = tl.sample(acc[0][q] * (1.0f / 81), key[0][q], io + q < g.ww && ko + j < g.hh);
                if (io < g.wp && ko + j < g.hh) {
                    typename BinQuad<B>::T u;
                    u.x = (B)b[0];
                    u.y = (B)b[1];
                    u.z = (B)b[2];
                    u.w = (B)b[3];
                    *reinterpret_cast<typename BinQuad<B>::T *>(out + (size_t)j * g.wp) = u;
                }
                /* The next row to where the loop's code reads it. */
#pragma unroll
                for (int i = 0; i + 1 < kNR; i++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        acc[i][q] = acc[i + 1][q];
                        key[i][q] = key[i + 1][q];
                    }
            }
        }
        tl.flush();
        __syncthreads();
        for (int b = tid; b < k.nb_bins; b += kBinNT) {
            const uint64_t T = (uint64_t)tally[b] + ((uint64_t)tally[k.nb_bins + b] << 17) +
                               ((uint64_t)tally[2 * k.nb_bins + b] << 34);
            if (!T)
                continue;
            tally[b] = tally[k.nb_bins + b] = tally[2 * k.nb_bins + b] = 0;
            /* T 2^-45 = T 2^19 in units of 2^-64. */
            const uint64_t f[3] = { (T << 19) & 0xffffffffu, (T >> 13) & 0xffffffffu, T >> 45 };
#pragma unroll
            for (int q = 0; q < 3; q++)
                if (f[q])
                    atomicAdd(reinterpret_cast<unsigned long long *>(&bins[b].sum[q]), (unsigned long long)f[q]);
        }
    }
    __syncthreads();
    for (int i = tid; i < k.nb_bins * g.win; i += kBinNT)
        if (hist[i])
            atomicAdd(&h1[(i / g.win) * kB1 + g.lo + i % g.win], hist[i]);
}

/* Level 2 or 3: the samples whose key agrees with their bin's prefix so
 * far, counted by their next 10 bits. A warp walks down a strip of
 * positions, four columns a lane, a lane of apron on either side, and forms
 * the high-pass again: 32 to 37 us at 5760x3240. Reading it back (112 MB with
 * its bin, not 19) took 22, and those 93 MB's pages 230 us a call to map and
 * to unmap. */
constexpr int kRefCols = 30 * 4, kRefWarps = 4;

template <int LEVEL, typename B>
__global__ void __launch_bounds__(32 * kRefWarps)
k_noise_refine(const CRAWKNoise k, const NoiseGrid g, const uint16_t *src, size_t pitch, const float *lut,
               const B *bidx, const uint2 *sel, uint32_t *hist, int nx, int seg)
{
    __shared__ uint32_t pre[CRAW_K_NOISE_MAX_BINS + 1];
    const int nb = k.nb_bins, w2 = k.width / 2, h2 = k.height / 2;
    craw_await_previous();
    craw_let_next_start();
    for (int b = threadIdx.x; b <= nb; b += 32 * kRefWarps)
        pre[b] = b < nb ? sel[b].x : kNone;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = blockIdx.x * kRefWarps + (threadIdx.x >> 5);
    const int py = wid & 1, sx = (wid >> 1) % nx, sy = (wid >> 1) / nx;
    const int k0 = sy * seg, k1 = min(k0 + seg, g.hh);
    if (k0 >= g.hh)
        return;
    const int io = sx * kRefCols + 4 * (lane - 1);
    const bool mine = lane >= 1 && lane <= 30 && io < g.wp;
    auto fetch = [&](int r) {                    /* plane row r, columns io + kR .. io + kR + 3 */
        return r < h2 ? plane_quad((const char *)src + (size_t)(2 * r + py) * pitch, io + kR, w2)
                      : make_uint4(0u, 0u, 0u, 0u);
    };
    float v[2][3][6];
    auto put = [&](uint4 raw) {
#pragma unroll
        for (int pl = 0; pl < 2; pl++) {
#pragma unroll
            for (int c = 0; c < 6; c++) {
                v[pl][0][c] = v[pl][1][c];
                v[pl][1][c] = v[pl][2][c];
            }
            const float4 x = plane_values(lut + (2 * py + pl) * 65536, raw, 16 * pl);
            v[pl][2][0] = __shfl_up_sync(0xffffffffu, x.w, 1);
            v[pl][2][1] = x.x;
            v[pl][2][2] = x.y;
            v[pl][2][3] = x.z;
            v[pl][2][4] = x.w;
            v[pl][2][5] = __shfl_down_sync(0xffffffffu, x.x, 1);
        }
    };
    uint4 raw[2] = { fetch(k0 + kR - 1), fetch(k0 + kR) };
    uint4 next = fetch(k0 + kR + 1);
    put(raw[0]);
    put(raw[1]);
#pragma unroll 1
    for (int ko = k0; ko < k1; ko++) {
        const uint4 now = next;
        next = fetch(ko + kR + 2);
        uint32_t b[2][4];
#pragma unroll
        for (int pl = 0; pl < 2; pl++) {
            using Q = typename BinQuad<B>::T;
            Q q;
            q.x = q.y = q.z = q.w = (B)nb;
            if (mine)
                q = *reinterpret_cast<const Q *>(bidx + ((size_t)(2 * py + pl) * g.hh + ko) * g.wp + io);
            b[pl][0] = q.x;
            b[pl][1] = q.y;
            b[pl][2] = q.z;
            b[pl][3] = q.w;
        }
        put(now);
#pragma unroll
        for (int pl = 0; pl < 2; pl++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t key = high_pass(v[pl][0], v[pl][1], v[pl][2], 1 + q);
                if ((key >> (LEVEL == 2 ? 20 : 10)) == pre[b[pl][q]])
                    atomicAdd(&hist[b[pl][q] * 1024 + ((LEVEL == 2 ? key >> 10 : key) & 1023u)], 1u);
            }
    }
}

/* One CTA per bin: the bucket of `hist` holding the bin's rank-th smallest
 * key (rank = count / 2 at level 1, then what is left of it inside the
 * chosen bucket); sel = (key prefix, remaining rank), a prefix that no key
 * has where the bin is empty. */
template <int LEVEL>
__global__ void __launch_bounds__(256) k_noise_select(const uint32_t *hist, uint2 *sel, CRAWKNoiseBin *bins)
{
    constexpr int PER = (LEVEL == 1 ? kB1 : kB2) / 256;
    static_assert(kB2 == kB3, "levels 2 and 3 alike");
    __shared__ uint32_t part[8];
    craw_await_previous();
    craw_let_next_start();
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint2 was = LEVEL == 1 ? make_uint2(0u, 0u) : sel[b];
    uint32_t h[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; j += 4)
        *reinterpret_cast<uint4 *>(h + j) = reinterpret_cast<const uint4 *>(hist)[((size_t)b * 256 + tid) * (PER / 4) + j / 4];
#pragma unroll
    for (int j = 0; j < PER; j++)
        sum += h[j];
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d)
            incl += o;
    }
    if (lane == 31)
        part[warp] = incl;
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        if (i == warp)
            incl += total;
        total += part[i];
    }
    if (LEVEL == 1 && tid == 0)
        bins[b].count = total;
    if (LEVEL == 1 ? total == 0 : was.x == kNone) {
        if (tid == 0) {
            sel[b] = make_uint2(kNone, 0u);
            bins[b].median = 0;
        }
        return;
    }
    const uint32_t rank = LEVEL == 1 ? total / 2 : was.y;
    if (rank >= incl || rank < incl - sum)
        return;
    uint32_t r = rank - (incl - sum), j = 0;
#pragma unroll
    for (int i = 0; i + 1 < PER; i++)
        if (j == (uint32_t)i && r >= h[i]) {
            r -= h[i];
            j++;
        }
    const uint32_t bucket = (uint32_t)(tid * PER) + j;
    const uint32_t prefix = LEVEL == 1 ? bucket : (was.x << 10) | bucket;
    sel[b] = make_uint2(prefix, r);
    if (LEVEL == 3)
        bins[b].median = prefix;
}

/* ------------------------------------------------ least trimmed squares */

/* The line through bins i and j, or false where the pair gives none. */
CRAW_DEV bool lts_line(const double *m, const double *v, int i, int j, double &a, double &b)
{
    const double dm = m[j] - m[i];
    if (dm < 1e-5)
        return false;
    a = (v[j] - v[i]) / dm;
    b = v[i] - a * m[i];
    return a > 0.0 && !(b < 0.0);
}

/* How far the root of a pair's float cost can be from that of its double
 * one. The root is the length of the vector of kept residuals, and the
 * least over the choices of what to keep, so it moves by no more than the
 * residuals do: each by the roundings of logf (a unit in the last place, at
 * most 2^-23 |log|) and its argument (3e-7), of lv and of the difference,
 * where |log| <= |lv| + |residual|: 1.8e-7 (|lv| + |residual|) + 3e-7; and
 * by those of the squares and of their sum (a tree of at most 21), 1e-6 of
 * it. Taken more than twice as large. */
CRAW_DEV float lts_slack(float root, float lmax, float rkeep)
{
    return 3e-6f * root + (5e-7f * lmax + 1e-6f) * rkeep;
}

constexpr int kLtsWarps = 4, kLtsPairs = 4;      /* pairs a warp: its line costs doubles, a lane a pair */

/* The root of every pair's trimmed cost in floats, root[i nb + j] (+inf: no
 * line), and the least upper bound of the least one. The keep smallest
 * squares by descent on the bits of the keep-th. */
template <int E>
__global__ void __launch_bounds__(32 * kLtsWarps)
k_noise_lts_float(const double *m, const double *v, const double *lv, int nb, int keep, float *root,
                  uint32_t *bound)
{
    craw_let_next_start();
    const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const int i = blockIdx.x, j0 = (blockIdx.y * kLtsWarps + warp) * kLtsPairs;
    if (j0 + kLtsPairs <= i + 1 || j0 >= nb)
        return;                                  /* whole warps only */
    float fm[E], fl[E], lmax = 0.0f;
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int t = lane + 32 * r;
        fm[r] = t < nb ? (float)m[t] : 0.0f;
        fl[r] = t < nb ? (float)lv[t] : 0.0f;
        lmax = fmaxf(lmax, fabsf(fl[r]));
    }
#pragma unroll
    for (int d = 16; d; d >>= 1)
        lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, d));
    double a = 0.0, b = 0.0;
    const int j = j0 + (lane & (kLtsPairs - 1));
    const bool line = j > i && j < nb && lts_line(m, v, i, j, a, b);
    const float fa = (float)a, fb = (float)b;
    float least = INFINITY;
    for (int p = 0; p < kLtsPairs; p++) {
        const int jp = j0 + p;
        if (jp <= i || jp >= nb)
            continue;
        const float pa = __shfl_sync(0xffffffffu, fa, p), pb = __shfl_sync(0xffffffffu, fb, p);
        float c = INFINITY;
        if (__shfl_sync(0xffffffffu, (int)line, p)) {
            uint32_t e[E];
#pragma unroll
            for (int r = 0; r < E; r++) {
                const float d = fl[r] - logf(pa * fm[r] + pb);
                e[r] = lane + 32 * r < nb ? __float_as_uint(d * d) : 0x7f800000u;
            }
            uint32_t T = 0;                      /* the keep-th smallest: the largest with fewer than keep below */
#pragma unroll 1
            for (int bit = 30; bit >= 0; bit--) {
                const uint32_t x = T | 1u << bit;
                int n = 0;
#pragma unroll
                for (int r = 0; r < E; r++)
                    n += __popc(__ballot_sync(0xffffffffu, e[r] < x));
                if (n < keep)
                    T = x;
            }
            int n = 0;
            float s = 0.0f;
#pragma unroll
            for (int r = 0; r < E; r++) {
                n += __popc(__ballot_sync(0xffffffffu, e[r] < T));
                s += e[r] < T ? __uint_as_float(e[r]) : 0.0f;
            }
#pragma unroll
            for (int d = 16; d; d >>= 1)
                s += __shfl_xor_sync(0xffffffffu, s, d);
            c = sqrtf(s + (float)(keep - n) * __uint_as_float(T));
        }
        if (lane == 0)
            root[(size_t)i * nb + jp] = c;
        least = fminf(least, c);
    }
    if (lane == 0 && least < INFINITY)
        atomicMin(bound, __float_as_uint(least + lts_slack(least, lmax, sqrtf((float)keep))));
}

/* The least of the double costs of the pairs that the floats leave in
 * question, the first of equals in (i, j) order. A warp looks at `span`
 * pairs, far apart (those in question come together); of one that may be the least it sorts the squared residuals
 * ascending in shared memory (bitonic; they are not negative, so their bits
 * sort as they do), and one lane adds the `keep` smallest in order. The
 * pairs that came this far gather in `found`; the last CTA to finish picks
 * from them. count: the pairs found, the CTAs done. */
constexpr int kLtsExactWarps = 8, kLtsSpan = 8, kLtsFew = 40;

__global__ void __launch_bounds__(32 * kLtsExactWarps)
k_noise_lts(const double *m, const double *v, const double *lv, int nb, int np2, int keep, int span,
            const float *root, const uint32_t *bound, ulonglong2 *found, uint32_t *count, int2 *best)
{
    __shared__ unsigned long long d2[kLtsExactWarps][CRAW_K_NOISE_MAX_BINS];
    __shared__ bool last;
    craw_await_previous();
    const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const int p0 = blockIdx.x * kLtsExactWarps + warp, step = gridDim.x * kLtsExactWarps;
    unsigned long long *w = d2[warp];
    float lmax = 0.0f;
    for (int t = lane; t < nb; t += 32)
        lmax = fmaxf(lmax, fabsf((float)lv[t]));
#pragma unroll
    for (int d = 16; d; d >>= 1)
        lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, d));
    bool maybe = false;
    const int mine = p0 + lane * step;
    if (lane < span && mine < nb * nb && mine / nb < mine % nb) {
        const float c = root[mine];
        maybe = c < INFINITY && c - lts_slack(c, lmax, sqrtf((float)keep)) <= __uint_as_float(*bound);
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, maybe); todo; todo &= todo - 1) {
        const int p = p0 + (__ffs(todo) - 1) * step;
        double a = 0.0, b = 0.0;
        if (!lts_line(m, v, p / nb, p % nb, a, b))
            continue;
        __syncwarp();
        for (int t = lane; t < np2; t += 32) {
            double d = INFINITY;
            if (t < nb) {
                d = lv[t] - log(a * m[t] + b);
                d = d * d;
            }
            w[t] = (unsigned long long)__double_as_longlong(d);
        }
        __syncwarp();
        for (int size = 2; size <= np2; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = lane; t < np2 / 2; t += 32) {
                    const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
                    const bool up = (lo & size) == 0;
                    const unsigned long long x = w[lo], y = w[hi];
                    if ((x > y) == up) {
                        w[lo] = y;
                        w[hi] = x;
                    }
                }
                __syncwarp();
            }
        if (lane == 0) {
            double c = 0.0;
            for (int t = 0; t < keep; t++)
                c += __longlong_as_double((long long)w[t]);
            found[atomicAdd(&count[0], 1u)] =
                make_ulonglong2((unsigned long long)__double_as_longlong(c), (unsigned long long)p);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        last = atomicAdd(&count[1], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || warp)
        return;
    __threadfence();
    const int n = (int)*(volatile uint32_t *)&count[0];
    const unsigned long long inf = 0x7ff0000000000000ull;
    unsigned long long c = inf, at = ~0ull;
    auto take = [&](unsigned long long x, unsigned long long q) {
        if (x < c || (x == c && q < at)) {
            c = x;
            at = q;
        }
    };
    for (int t = lane; t < n; t += 32) {
        const volatile unsigned long long *f = reinterpret_cast<const volatile unsigned long long *>(found + t);
        take(f[0], f[1]);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, c, d), q = __shfl_xor_sync(0xffffffffu, at, d);
        take(x, q);
    }
    if (lane == 0)
        *best = c < inf ? make_int2((int)at / nb, (int)at % nb) : make_int2(-1, -1);
}

/* The two bin-index widths' launches. */
template <typename B>
int noise_bins(const CRAWKNoise *k, const uint16_t *src, size_t pitch, char *base, const Layout &L,
               CRAWKNoiseBin *bins, cudaStream_t s)
{
    const NoiseGrid g = noise_grid(k->width, k->height, k->nb_bins);
    const float *lut = reinterpret_cast<const float *>(base + L.lut);
    uint32_t *h1 = reinterpret_cast<uint32_t *>(base + L.h1);
    uint32_t *h2 = reinterpret_cast<uint32_t *>(base + L.h2);
    uint32_t *h3 = reinterpret_cast<uint32_t *>(base + L.h3);
    uint2 *sel = reinterpret_cast<uint2 *>(base + L.sel);
    B *bidx = reinterpret_cast<B *>(base + L.bidx);
    static std::atomic<uint64_t> attr_done{ 0 };
    constexpr size_t most = 2 * kPH * kPW * sizeof(float) + 65536 + 3 * CRAW_K_NOISE_MAX_BINS * sizeof(uint32_t);
    if (craw_smem_attr(k_noise_bin<B>, most, attr_done) < 0)
        return -5;
    const size_t smem = 2 * kPH * kPW * sizeof(float) + (size_t)k->nb_bins * (g.win + 3) * sizeof(uint32_t);
    const int items = 2 * g.ntx * g.nty, room = 2 * 152;
    /* Each ready to start when the one before it ends (2 to 5 %
     * of an estimate at 5760x3240). */
    if (craw_launch_early(k_noise_bin<B>, items < room ? items : room, kBinNT, smem, true, s, *k, g, src, pitch, lut,
                          h1, bidx, bins) < 0 ||
        craw_launch_early(k_noise_select<1>, k->nb_bins, 256, 0, true, s, h1, sel, bins) < 0)
        return -5;
    /* Segments of about one wave of 28 warps an SM, at least 8 rows. */
    const int nx = (g.ww + kRefCols - 1) / kRefCols, nseg = 152 * 28 / (2 * nx) > 1 ? 152 * 28 / (2 * nx) : 1;
    const int seg = (g.hh + nseg - 1) / nseg < 8 ? 8 : (g.hh + nseg - 1) / nseg;
    const int warps = 2 * nx * ((g.hh + seg - 1) / seg), ctas = (warps + kRefWarps - 1) / kRefWarps;
    if (craw_launch_early(k_noise_refine<2, B>, ctas, 32 * kRefWarps, 0, true, s, *k, g, src, pitch, lut, bidx, sel,
                          h2, nx, seg) < 0 ||
        craw_launch_early(k_noise_select<2>, k->nb_bins, 256, 0, true, s, h2, sel, bins) < 0 ||
        craw_launch_early(k_noise_refine<3, B>, ctas, 32 * kRefWarps, 0, true, s, *k, g, src, pitch, lut, bidx, sel,
                          h3, nx, seg) < 0)
        return -5;
    return craw_launch_early(k_noise_select<3>, k->nb_bins, 256, 0, true, s, h3, sel, bins);
}

} // namespace

extern "C" size_t craw_k_noise_scratch(int32_t width, int32_t height, int32_t nb_bins)
{
    return layout(width, height, nb_bins).total;
}

extern "C" int craw_k_noise_bins(const CRAWKNoise *k, const uint16_t *src, size_t src_pitch, void *scratch,
                                 CRAWKNoiseBin *bins, cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    const Layout L = layout(k->width, k->height, k->nb_bins);
    char *base = static_cast<char *>(scratch);
    NoiseSite site;
    for (int i = 0; i < 4; i++) {
        const float range = k->white[i] - k->black[i];          /* float, as the reference */
        site.black[i] = (double)k->black[i];
        site.range[i] = (double)range;
        site.rcp[i] = 1.0 / (double)range;
    }
    if (cudaMemsetAsync(base + L.h1, 0, L.sel - L.h1, s) != cudaSuccess ||
        cudaMemsetAsync(bins, 0, (size_t)k->nb_bins * sizeof(CRAWKNoiseBin), s) != cudaSuccess)
        return -5;
    k_noise_lut<<<dim3(65536 / 256, 4), 256, 0, s>>>(site, reinterpret_cast<float *>(base + L.lut));
    if (cudaGetLastError() != cudaSuccess)
        return -5;
    return bin_bytes(k->nb_bins) == 1 ? noise_bins<uint8_t>(k, src, src_pitch, base, L, bins, s)
                                      : noise_bins<uint16_t>(k, src, src_pitch, base, L, bins, s);
}

extern "C" size_t craw_k_noise_lts_scratch(int32_t nb)
{
    return (size_t)nb * nb * (sizeof(ulonglong2) + sizeof(float)) + 256;
}

extern "C" int craw_k_noise_lts(const double *m, const double *v, const double *lv, int32_t nb, int32_t keep,
                                void *scratch, int32_t best[2], cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    if (nb < 2 || nb > CRAW_K_NOISE_MAX_BINS)
        return -22;
    int np2 = 32;
    while (np2 < nb)
        np2 <<= 1;
    /* The bound (from above every finite root, 0x7f7f7f7f: 3.4e38), the
     * counts, the found pairs, the roots. */
    uint32_t *bound = static_cast<uint32_t *>(scratch), *count = bound + 1;
    ulonglong2 *found = reinterpret_cast<ulonglong2 *>(static_cast<char *>(scratch) + 256);
    float *root = reinterpret_cast<float *>(found + (size_t)nb * nb);
    if (cudaMemsetAsync(bound, 0x7f, 4, s) != cudaSuccess || cudaMemsetAsync(count, 0, 8, s) != cudaSuccess)
        return -5;
    const int per = kLtsWarps * kLtsPairs;
    const dim3 grid(nb, (nb + per - 1) / per);
    /* A few bins' pairs are all evaluated in doubles at once, a warp each:
     * 8 bins 13.5 us (21.6 through the floats), 32 bins 20.8 (23.8), 40 bins
     * 26.0 (26.1), 48 bins 30.1 (26.3), 64 bins 40.4 (27.0). */
    const bool few = nb <= kLtsFew;
    if (few) {
        if (cudaMemsetAsync(root, 0, (size_t)nb * nb * sizeof(float), s) != cudaSuccess)
            return -5;
    } else if (nb <= 128)
        k_noise_lts_float<4><<<grid, 32 * kLtsWarps, 0, s>>>(m, v, lv, nb, keep, root, bound);
    else
        k_noise_lts_float<16><<<grid, 32 * kLtsWarps, 0, s>>>(m, v, lv, nb, keep, root, bound);
    if (cudaGetLastError() != cudaSuccess)
        return -5;
    const int span = few ? 1 : kLtsSpan, cta = span * kLtsExactWarps;
    return craw_launch_early(k_noise_lts, (nb * nb + cta - 1) / cta, 32 * kLtsExactWarps, 0, !few, s, m, v, lv, nb,
                             np2, keep, span, root, bound, found, count, reinterpret_cast<int2 *>(best));
}
