/* A CUDA runtime without a GPU, preloaded in place of libcudart by test_host_launches.py.
 * Device memory is host memory, copies and fills work, kernels are not run; every launch
 * is checked against what the real runtime refuses (grid and block sizes, dynamic shared
 * memory beyond 48 KB without the function's opt-in on the current device) and written to
 * the file FAKE_CUDA_LOG as "<device> <kernel> <status> <dynamic shared memory> <opt-in>".
 * fake_fail_in: launches until one fails (-1: none does); fake_memory: bytes the device has;
 * fake_in_use: bytes taken. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define API __attribute__((visibility("default")))
enum { DEVICES = 2, FUNCS = 4096 };

static struct { const void *fn; const char *name; int smem[DEVICES]; } funcs[FUNCS];
static int nfuncs, device;
static cudaError_t last;
API int fake_fail_in = -1;
API size_t fake_memory = (size_t)-1, fake_in_use;

static cudaError_t out(cudaError_t e)
{
    if (e != cudaSuccess) last = e;
    return e;
}

static int find(const void *fn)
{
    for (int i = 0; i < nfuncs; i++)
        if (funcs[i].fn == fn) return i;
    return -1;
}

/* what the compiler's host code calls */
API void **__cudaRegisterFatBinary(void *b) { return (void **)b; }
API void __cudaRegisterFatBinaryEnd(void **b) { (void)b; }
API void __cudaUnregisterFatBinary(void **b) { (void)b; }
API void __cudaRegisterVar(void **b, char *host, char *dev, const char *name, int ext, size_t size, int c, int g)
{
    (void)b, (void)host, (void)dev, (void)name, (void)ext, (void)size, (void)c, (void)g;
}
API void __cudaRegisterFunction(void **b, const char *host, char *dev, const char *name, int limit, void *tid, void *bid,
                                void *bdim, void *gdim, int *wsize)
{
    (void)b, (void)dev, (void)limit, (void)tid, (void)bid, (void)bdim, (void)gdim, (void)wsize;
    if (nfuncs < FUNCS) {
        funcs[nfuncs].fn = host;
        funcs[nfuncs++].name = name;
    }
}
API cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn)
{
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
API unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, void *s)
{
    (void)g, (void)b, (void)m, (void)s;
    abort(); /* no <<<>>> launches */
}
API cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s)
{
    (void)g, (void)b, (void)m, (void)s;
    abort();
}
API cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **args, size_t m, cudaStream_t s)
{
    (void)k, (void)g, (void)b, (void)args, (void)m, (void)s;
    abort();
}

static cudaError_t launch(const void *fn, dim3 g, dim3 b, size_t smem)
{
    static FILE *log;
    const int f = find(fn);
    cudaError_t e = cudaSuccess;
    if (f < 0) e = cudaErrorInvalidDeviceFunction;
    else if (!g.x || !g.y || !g.z || g.x > 0x7FFFFFFFu || g.y > 65535 || g.z > 65535) e = cudaErrorInvalidConfiguration;
    else if (!b.x || !b.y || !b.z || (uint64_t)b.x * b.y * b.z > 1024) e = cudaErrorInvalidConfiguration;
    else if (smem > 48 * 1024 && smem > (size_t)funcs[f].smem[device]) e = cudaErrorInvalidValue;
    else if (fake_fail_in == 0) e = cudaErrorLaunchOutOfResources;
    if (fake_fail_in >= 0) fake_fail_in--;
    if (!log) log = fopen(getenv("FAKE_CUDA_LOG"), "w");
    fprintf(log, "%d %s %d %zu %d\n", device, f < 0 ? "?" : funcs[f].name, (int)e, smem, f < 0 ? 0 : funcs[f].smem[device]);
    fflush(log);
    return out(e);
}
API cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args)
{
    (void)args;
    return launch(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
API cudaError_t cudaLaunchCooperativeKernel(const void *fn, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t s)
{
    (void)args, (void)s;
    return launch(fn, g, b, smem);
}
API cudaError_t cudaFuncSetAttribute(const void *fn, enum cudaFuncAttribute a, int v)
{
    const int f = find(fn);
    if (f < 0) return out(cudaErrorInvalidDeviceFunction);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) funcs[f].smem[device] = v;
    return cudaSuccess;
}

/* a device reset takes the functions' opt-ins with it */
API void fake_reset(void)
{
    for (int i = 0; i < nfuncs; i++) memset(funcs[i].smem, 0, sizeof funcs[i].smem);
}

/* memory: each block holds its start and size before the address given out */
static cudaError_t take(void **p, size_t bytes)
{
    if (fake_in_use + bytes > fake_memory) return out(cudaErrorMemoryAllocation);
    char *m = calloc(1, bytes + 512);
    if (!m) return out(cudaErrorMemoryAllocation);
    uintptr_t a = ((uintptr_t)m + 256 + 255) & ~(uintptr_t)255;
    ((void **)a)[-1] = m;
    ((size_t *)a)[-2] = bytes;
    fake_in_use += bytes;
    *p = (void *)a;
    return cudaSuccess;
}
static cudaError_t give(void *p)
{
    if (!p) return cudaSuccess;
    fake_in_use -= ((size_t *)p)[-2];
    free(((void **)p)[-1]);
    return cudaSuccess;
}
API cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
API cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) { (void)s; return take(p, n); }
API cudaError_t cudaFree(void *p) { return give(p); }
API cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { (void)s; return give(p); }
API cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
    (void)k;
    memmove(d, s, n);
    return cudaSuccess;
}
API cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
API cudaError_t cudaMemset(void *d, int v, size_t n)
{
    memset(d, v, n);
    return cudaSuccess;
}
API cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s)
{
    (void)s;
    return cudaMemset(d, v, n);
}

/* the rest succeeds */
API cudaError_t cudaGetLastError(void)
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
API const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "error of the fake runtime"; }
API cudaError_t cudaSetDevice(int d)
{
    if (d < 0 || d >= DEVICES) return out(cudaErrorInvalidDevice);
    device = d;
    return cudaSuccess;
}
API cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
API cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
API cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int d) { (void)d; *p = (cudaMemPool_t)16; return cudaSuccess; }
API cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, enum cudaMemPoolAttr a, void *v) { (void)p, (void)a, (void)v; return cudaSuccess; }
API cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)16; return cudaSuccess; }
API cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
API cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
API cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e, (void)s; return cudaSuccess; }
API cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
API cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a, (void)b; *ms = 1.0f; return cudaSuccess; }
API cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)32; return cudaSuccess; }
API cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
API cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
API cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) { (void)s; *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
API cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s, (void)m; return cudaSuccess; }
API cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)16; return cudaSuccess; }
API cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) { (void)g, (void)f; *x = (cudaGraphExec_t)16; return cudaSuccess; }
API cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t *n, size_t *c) { (void)g, (void)n; *c = 0; return cudaSuccess; }
API cudaError_t cudaGraphNodeGetType(cudaGraphNode_t n, enum cudaGraphNodeType *t) { (void)n; *t = cudaGraphNodeTypeKernel; return cudaSuccess; }
API cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x, (void)s; return cudaSuccess; }
API cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
API cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { (void)x; return cudaSuccess; }
API cudaError_t cudaGetSymbolAddress(void **p, const void *s) { (void)s; static char m[1 << 26]; *p = m; return cudaSuccess; }
API cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl)
{
    (void)f, (void)b, (void)s, (void)fl;
    *n = 4;
    return cudaSuccess;
}
