/* cudart.c — the CUDA runtime calls of the host code, on host memory: no device, no kernels, one
 * stream that runs everything at once. For tests of what the host does when a call fails or a
 * pass does not fit; fake_alloc_limit makes larger device allocations fail. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

static size_t g_limit; /* bytes (0: none) */
static long g_allocs;  /* device and page-locked allocations made */
static cudaError_t g_last;
static int g_locked;   /* all host memory is page-locked */
static char g_token[16];

void fake_alloc_limit(size_t bytes) { g_limit = bytes; }
void fake_page_locked(int on) { g_locked = on; }
long fake_allocs(void) { return g_allocs; }

static cudaError_t fail(cudaError_t e)
{
    g_last = e;
    return e;
}

cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "a failure of the test's"; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d == 0 ? cudaSuccess : fail(cudaErrorInvalidDevice); }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 152; return cudaSuccess; }

cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t s)
{
    (void)s;
    if (g_limit && bytes > g_limit) return fail(cudaErrorMemoryAllocation);
    g_allocs++;
    *p = aligned_alloc(256, (bytes + 255) & ~(size_t)255);
    return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { (void)s; free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t bytes)
{
    g_allocs++;
    *p = malloc(bytes ? bytes : 1);
    return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)k;
    (void)st;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, 0); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s) { (void)s; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol) { *p = (void *)symbol; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p)
{
    memset(a, 0, sizeof(*a)); /* ordinary host memory */
    if (g_locked) {
        a->type = cudaMemoryTypeHost;
        a->devicePointer = a->hostPointer = (void *)p;
    }
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)g_token; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = (cudaEvent_t)g_token; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 0.0f; return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)g_token; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f)
{
    (void)g;
    (void)f;
    *x = (cudaGraphExec_t)g_token;
    return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t x, cudaGraph_t g, cudaGraphExecUpdateResultInfo *i)
{
    (void)x;
    (void)g;
    (void)i;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { (void)x; return cudaSuccess; }

/* what an object of nvcc's registers with the runtime when it is loaded */
void **__cudaRegisterFatBinary(void *b) { (void)b; return (void **)g_token; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int x, size_t s, int c, int g)
{
    (void)h, (void)v, (void)a, (void)n, (void)x, (void)s, (void)c, (void)g;
}
