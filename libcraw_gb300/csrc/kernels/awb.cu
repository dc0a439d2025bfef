/*
 * The AWB histogram's way to the host: the frame's three 128 x 128
 * histograms (count, sum of min(g, 0.5), sum of g^4; reference
 * lib/awb.c:287-291), the count of deferred blocks and the first of them,
 * from the device slot the develop kernels filled straight into its pinned
 * host copy, and the device slot back to zeros for its next frame.
 *
 * Bound: its launch, which the develop kernel lets start early (a 1920x1080
 * bilinear frame: 16.4 us, 18.9 with a plain launch). A fill before the frame and a copy after it took 9 to
 * 13 us of a frame's device time (the 256 KB copy alone 7 to 11); this one
 * kernel, 4.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace {

constexpr int kVecs = 3 * 128 * 128 / 4;       /* 16-byte pieces of the histograms */
constexpr int kThreads = 256;

/* One piece a thread; thread i also takes deferred block i. `head`: the
 * count, and a ticket that tells the last CTA to zero it. */
__global__ void __launch_bounds__(kThreads)
k_awb_publish(uint4 *hist, uint32_t *head, const uint4 *deferred, uint4 *host_hist, uint32_t *host_head,
              uint4 *host_deferred)
{
    craw_await_previous();
    const int i = blockIdx.x * kThreads + threadIdx.x;
    const uint32_t n = *(volatile uint32_t *)head;
    host_hist[i] = hist[i];
    hist[i] = make_uint4(0u, 0u, 0u, 0u);
    if (i < CRAW_K_AWB_DEFER_MAX && (uint32_t)i < n)
        host_deferred[i] = deferred[i];
    if (i == 0)
        host_head[0] = n;
    __syncthreads();                            /* the CTA's threads have read the count */
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&head[1], 1u) == gridDim.x - 1) {
            head[0] = 0;
            head[1] = 0;
        }
    }
}

static_assert(kVecs % kThreads == 0 && CRAW_K_AWB_DEFER_MAX <= kVecs, "a thread a piece and a block");
static_assert(sizeof(CRAWKAwbDeferred) == 16, "a deferred block is one piece");

} // namespace

extern "C" int craw_k_awb_publish(const CRAWKAwbOut *awb, void *host_hist, void *host_head, void *host_deferred,
                                  cudaStream_t s)
{
    if (craw_launch_ready() < 0)
        return -5;
    return craw_launch_early(k_awb_publish, kVecs / kThreads, kThreads, 0, true, s,
                             reinterpret_cast<uint4 *>(awb->hist), awb->nb_deferred,
                             reinterpret_cast<const uint4 *>(awb->deferred), static_cast<uint4 *>(host_hist),
                             static_cast<uint32_t *>(host_head), static_cast<uint4 *>(host_deferred));
}
