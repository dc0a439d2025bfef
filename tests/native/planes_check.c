/*
 * A pipeline's optional planes (alloc_planes of csrc/host/pipeline.c) on
 * failing calls: the allocator, the wait after it and the runtime's last
 * error are this file's. Built as a shared library with lazy binding; what
 * else pipeline.c calls is not reached.
 */
#include "../../libcraw_gb300/csrc/host/pipeline.c"

int craw_forced_denoise_shape = -1;
float craw_round_scale;

static int alloc_ret, sync_ret, live;
static cudaError_t pending;
static float buffer;

int craw_dev_alloc(CRAWContext *ctx, void **ptr, size_t bytes)
{
    *ptr = NULL;
    if (alloc_ret < 0)
        return alloc_ret;
    live++;
    *ptr = &buffer;
    return 0;
}

void craw_dev_free(CRAWContext *ctx, void *ptr)
{
    live -= ptr != NULL;
}

int craw_dev_sync(CRAWContext *ctx)
{
    return sync_ret;
}

size_t craw_k_denoise_planes(int32_t pw, int32_t ph)
{
    return 8 * sizeof(float) * (size_t)pw * ph;
}

cudaError_t cudaPeekAtLastError(void)
{
    return pending;
}

cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = pending;
    pending = cudaSuccess;
    return e;
}

/* out: what it returned, whether there are planes, buffers allocated and not
 * freed, the error left pending. */
__attribute__((visibility("default"))) void planes_check(int alloc, int sync, int error, int out[4])
{
    CRAWPipeline p = { 0 };
    float *planes = NULL;
    alloc_ret = alloc;
    sync_ret = sync;
    pending = (cudaError_t)error;
    live = 0;
    out[0] = alloc_planes(&p, &planes);
    out[1] = planes != NULL;
    out[2] = live;
    out[3] = (int)pending;
}
