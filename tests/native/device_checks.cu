/*
 * Device arithmetic that stands in for a division, against the division: each
 * check counts the inputs whose results differ in any bit. Compiled with the
 * kernels' own sources and the flags they are built with.
 */
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>

#include "../../libcraw_gb300/csrc/kernels/common.cuh"

namespace hl {
#include "../../libcraw_gb300/csrc/kernels/highlight.cu"
}
namespace nz {
#include "../../libcraw_gb300/csrc/kernels/noise.cu"
}

namespace {

__device__ bool differ(float a, float b)
{
    return __float_as_uint(a) != __float_as_uint(b);
}

/* F(bits) over the float bit patterns first .. last. */
template <typename F>
__global__ void k_count(uint32_t first, uint32_t last, F f, unsigned long long *bad)
{
    unsigned long long n = 0;
    for (uint64_t i = first + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= last;
         i += (uint64_t)gridDim.x * blockDim.x)
        n += f(__uint_as_float((uint32_t)i));
    if (n)
        atomicAdd(bad, n);
}

struct Reciprocal {
    __device__ bool operator()(float x) const { return differ(craw_rcp(x), 1.0f / x); }
};

struct GamutQuotient {
    float scl, iscl;
    __device__ bool operator()(float x) const { return differ(craw_gamut_quotient(x, scl, iscl), __fdiv_rn(x, scl)); }
};

/* The compression by divisions and the fast power. */
__device__ void gamut_compress(const CRAWKColor &c, float o[3])
{
    const float ach = fmaxf(o[0], fmaxf(o[1], o[2]));
    if (ach == 0.0f)
        return;
    const float mag = fabsf(ach), inv_mag = 1.0f / mag;
    for (int i = 0; i < 3; i++) {
        float d = (ach - o[i]) * inv_mag;
        if (d < c.gc_thr[i])
            continue;
        const float nd = __fdiv_rn(d - c.gc_thr[i], c.gc_scl[i]), p = __powf(nd, c.gc_pwr);
        d = c.gc_thr[i] + c.gc_scl[i] * nd * __powf(1.0f + p, -c.gc_inv_pwr);
        o[i] = ach - d * mag;
    }
}

/* A pixel of each x: its colours x times small and large ratios, and one of
 * zeros, infinities, NaN and x. */
struct Gamut {
    CRAWKColor c;
    __device__ bool operator()(float x) const
    {
        const float ratio[8] = { 1.0f, 0.9f, 0.19f, 0.05f, 0.0f, -0.2f, -3.0f, -1e4f };
        const float odd[5] = { 0.0f, -0.0f, INFINITY, -INFINITY, NAN };
        uint32_t h = __float_as_uint(x) * 2654435761u;
        float a[3], b[3];
        for (int i = 0; i < 3; i++, h = h * 747796405u + 2891336453u) {
            a[i] = x * ratio[(h >> 16) & 7] * (1.0f + (float)(h >> 8 & 0xff) / 4096.0f);
            if (!(h >> 20 & 15))
                a[i] = odd[(h >> 24) % 5];
            b[i] = a[i];
        }
        craw_gamut_compress(c, a);
        gamut_compress(c, b);
        for (int i = 0; i < 3; i++)
            if (differ(a[i], b[i]) && !(isnan(a[i]) && isnan(b[i])))
                return true;
        return false;
    }
};

struct ClipRamp {
    __device__ bool operator()(float v) const
    {
        float t = v <= hl::kULo ? 0.0f : __fdiv_rn(v - hl::kULo, hl::kUHi - hl::kULo);
        t = t < 0.0f ? 0.0f : (t > 1.0f ? 1.0f : t);
        return differ(hl::smooth(v), t * t * (3.0f - 2.0f * t));
    }
};

__global__ void k_lut_differs(const __grid_constant__ nz::NoiseSite n, const float *lut, unsigned long long *bad)
{
    const int s = blockIdx.y, raw = blockIdx.x * 256 + threadIdx.x;
    if (differ(lut[s * 65536 + raw], (float)(((double)raw * (1.0 / 65535.0) - n.black[s]) / n.range[s])))
        atomicAdd(bad, 1ull);
}

/* Counts, or -1 on a CUDA error. */
template <typename Launch>
long long counted(Launch launch)
{
    unsigned long long *bad = nullptr, n = 0;
    if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess)
        return -1;
    bool ok = cudaMemset(bad, 0, sizeof(*bad)) == cudaSuccess;
    if (ok)
        launch(bad);
    ok = ok && cudaMemcpy(&n, bad, sizeof(n), cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(bad);
    return ok ? (long long)n : -1;
}

template <typename F>
long long over(uint32_t first, uint32_t last, F f)
{
    return counted([&](unsigned long long *bad) { k_count<<<152 * 8, 256>>>(first, last, f, bad); });
}

} // namespace

#define CHECK extern "C" __attribute__((visibility("default"))) long long

/* The floats whose bits are first .. last. */
CHECK check_reciprocal(uint32_t first, uint32_t last) { return over(first, last, Reciprocal{}); }

/* Every float from 2^-30 to 2^100. */
CHECK check_gamut_quotient(float scl) { return over(97u << 23, 227u << 23, GamutQuotient{ scl, 1.0f / scl }); }

/* The same, as pixels, with the channels' thresholds and scales. */
CHECK check_gamut_compress(uint32_t first, uint32_t last, const float thr[3], const float scl[3], float pwr)
{
    Gamut g = {};
    for (int i = 0; i < 3; i++) {
        g.c.gc_thr[i] = thr[i];
        g.c.gc_scl[i] = scl[i];
        g.c.gc_iscl[i] = 1.0f / scl[i];
    }
    g.c.gc_pwr = pwr;
    g.c.gc_inv_pwr = (float)(1.0 / 1.2);
    return over(first, last, g);
}

/* Every float but NaN, of either sign. */
CHECK check_clip_ramp()
{
    const long long p = over(0u, 0x7f800000u, ClipRamp{}), n = over(0x80000000u, 0xff800000u, ClipRamp{});
    return p < 0 || n < 0 ? -1 : p + n;
}

/* Every 16-bit code at four sites' levels. */
CHECK check_noise_lut(const float black[4], const float white[4])
{
    nz::NoiseSite n;
    for (int s = 0; s < 4; s++) {
        const float range = white[s] - black[s];
        n.black[s] = (double)black[s];
        n.range[s] = (double)range;
        n.rcp[s] = 1.0 / (double)range;
    }
    float *lut = nullptr;
    if (cudaMalloc(&lut, 4 * 65536 * sizeof(float)) != cudaSuccess)
        return -1;
    const long long r = counted([&](unsigned long long *bad) {
        nz::k_noise_lut<<<dim3(256, 4), 256>>>(n, lut);
        k_lut_differs<<<dim3(256, 4), 256>>>(n, lut, bad);
    });
    cudaFree(lut);
    return r;
}
