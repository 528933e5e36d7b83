/*
 * A CUDA runtime in host memory for tests of the library's host code (sgrid.c,
 * sgrid_batch.c) without a GPU: allocations are malloc, copies are memcpy, kernels
 * do nothing.  A test can make the k-th allocation from now fail, mark a stream
 * as capturing, and read how much is allocated and what touched the legacy
 * default stream.
 */
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define EXPORT __attribute__((visibility("default")))

static long g_live, g_allocs, g_frees, g_fail_at = -1, g_legacy, g_waits, g_pool_live;
static cudaStream_t g_capturing;
static enum cudaStreamCaptureMode g_mode = cudaStreamCaptureModeGlobal;
static long g_unsafe; /* calls that a capturing stream forbids, made in the global mode */

EXPORT long fake_live(void) { return g_live; }
EXPORT long fake_pool_live(void) { return g_pool_live; }
EXPORT long fake_allocs(void) { return g_allocs; }
EXPORT long fake_frees(void) { return g_frees; }
EXPORT long fake_legacy(void) { return g_legacy; }
EXPORT long fake_waits(void) { return g_waits; }
EXPORT long fake_unsafe(void) { return g_unsafe; }
/* the k-th allocation from now (0: the next) fails, once; -1: none */
EXPORT void fake_fail(long k) { g_fail_at = k < 0 ? -1 : g_allocs + k; }
EXPORT void fake_capture(void *stream) { g_capturing = (cudaStream_t)stream; }

static void unsafe(void)
{
    if (g_capturing && g_mode == cudaStreamCaptureModeGlobal) g_unsafe++;
}
static void on(cudaStream_t st) { g_legacy += st == 0; }

static cudaError_t take(void **p, size_t bytes)
{
    if (g_allocs++ == g_fail_at) {
        *p = NULL;
        return cudaErrorMemoryAllocation;
    }
    *p = malloc(bytes ? bytes : 1);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaMalloc(void **p, size_t bytes)
{
    cudaError_t e;
    unsafe();
    if ((e = take(p, bytes)) == cudaSuccess) g_live++;
    return e;
}
cudaError_t cudaFree(void *p)
{
    unsafe();
    if (p) g_live--, g_frees++;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t st)
{
    cudaError_t e = take(p, bytes);
    (void)pool, (void)st;
    if (e == cudaSuccess) g_pool_live++;
    return e;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t st)
{
    (void)st;
    g_pool_live--;
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const struct cudaMemPoolProps *props)
{
    (void)props;
    *pool = (cudaMemPool_t)&g_pool_live;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) { return (void)p, (void)a, (void)v, cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) { return (void)p, (void)keep, cudaSuccess; }

cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)k;
    on(st);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
    unsafe();
    g_waits++;
    return cudaMemcpyAsync(d, s, n, k, 0);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st)
{
    on(st);
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, 0); }
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    unsafe();
    on(st);
    g_waits++;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *st, unsigned f)
{
    (void)f;
    *st = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st)
{
    free(st);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t st, enum cudaStreamCaptureStatus *s)
{
    *s = st && st == g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode *m)
{
    enum cudaStreamCaptureMode was = g_mode;
    g_mode = *m;
    *m = was;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned f) { return (void)st, (void)e, (void)f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t st, enum cudaStreamCaptureMode m) { return (void)st, (void)m, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t st, cudaGraph_t *g)
{
    (void)st;
    *g = (cudaGraph_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f)
{
    (void)g, (void)f;
    *x = (cudaGraphExec_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return free(x), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t st) { return (void)x, (void)st, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f)
{
    (void)f;
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { return (void)e, (void)st, cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return (void)e, cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b)
{
    (void)a, (void)b;
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) { return (void)d, cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorName(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
const char *cudaGetErrorString(cudaError_t e) { return cudaGetErrorName(e); }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
    (void)p;
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *s, void **f, unsigned v, unsigned long long fl,
                                             enum cudaDriverEntryPointQueryResult *q)
{
    (void)s, (void)v, (void)fl, (void)q;
    *f = NULL;
    return cudaErrorNotSupported;
}

/* ---- the launchers with a result; the test adds empty ones for the rest ---- */
static int64_t g_launches;
void sgk_count(int n) { g_launches += n; }
int64_t sgk_launches(void) { return g_launches; }
int sgk_num_sms(void) { return 148; }
int64_t sgk_chain_smem_bytes(int64_t cap, int eb) { return 2 * cap * eb <= 200 * 1024 ? 2 * cap * eb : -1; }
int64_t sgk_small_smem_bytes(int64_t cap, int eb) { return 8 * cap * eb <= 200 * 1024 ? 8 * cap * eb : -1; }
int64_t sgk_sort_scratch_bytes(int64_t m, int d) { return (void)d, 4 * m + 4096; }
int sgk_batch_sort_bits(int64_t m, int d) { return (void)m, (void)d, 4; }
int64_t sgk_batch_sort_scratch_bytes(int64_t p, int64_t b) { return 4 * (p + b) + 4096; }
