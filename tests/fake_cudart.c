/* A stand-in for the CUDA runtime, for tests of the library's host code without a
 * GPU: device memory is host memory, kernels are not run, and every launch is checked
 * and counted as the runtime would.  What it models:
 *   - several devices; a kernel's dynamic shared-memory limit belongs to one device,
 *     and a launch above it (48 KB where it was never raised) is refused;
 *   - the last error of a thread, which cudaGetLastError clears;
 *   - chosen kernels, limits and allocations being refused (the fake_* calls). */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

enum { MAXF = 512, MAXD = 8, MAXA = 4096 };
static struct { const void *host; const char *name; int limit[MAXD]; int runs[MAXD]; int refused[MAXD]; } fn[MAXF];
static struct { void *p; size_t bytes; } mem[MAXA];
static int nfn, clusters = 1000;
static size_t capacity = (size_t)256 << 30, used, largest;
static char no_launch[128], no_limit[128], no_cluster[128];
static __thread int device;
static __thread cudaError_t last;

static cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
static int find(const void *host)
{
    for (int i = 0; i < nfn; ++i) if (fn[i].host == host) return i;
    abort();
}
static int named(int f, const char *part) { return part[0] && strstr(fn[f].name, part); }

/* what the tests set and read */
void fake_clusters(int n) { clusters = n; }
void fake_capacity(size_t n) { capacity = n; }
size_t fake_used(void) { return used; }
void fake_refuse_launch(const char *part) { snprintf(no_launch, sizeof no_launch, "%s", part); }
void fake_refuse_limit(const char *part) { snprintf(no_limit, sizeof no_limit, "%s", part); }
void fake_refuse_cluster(const char *part) { snprintf(no_cluster, sizeof no_cluster, "%s", part); }
size_t fake_largest_alloc(void) { size_t n = largest; largest = 0; return n; }
static int sum(const char *part, int dev, int refused)
{
    int n = 0;
    for (int i = 0; i < nfn; ++i)
        if (named(i, part)) n += refused ? fn[i].refused[dev] : fn[i].runs[dev];
    return n;
}
int fake_runs(const char *part, int dev) { return sum(part, dev, 0); }
int fake_refused(const char *part, int dev) { return sum(part, dev, 1); }

/* registration and launches */
void **__cudaRegisterFatBinary(void *p) { (void)p; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *d, const char *n, int e, size_t s, int c, int g)
{
    (void)h; (void)v; (void)d; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int t, void *a, void *b, void *c,
                            void *d, int *w)
{
    (void)h; (void)dev; (void)t; (void)a; (void)b; (void)c; (void)d; (void)w;
    if (nfn == MAXF) abort();
    fn[nfn].host = host;
    fn[nfn++].name = name;
}
static __thread struct { struct dim3 grid, block; size_t smem; void *stream; } cfg;
unsigned __cudaPushCallConfiguration(struct dim3 grid, struct dim3 block, size_t smem, void *stream)
{
    cfg.grid = grid; cfg.block = block; cfg.smem = smem; cfg.stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(struct dim3 *grid, struct dim3 *block, size_t *smem, void *stream)
{
    *grid = cfg.grid; *block = cfg.block; *smem = cfg.smem; *(void **)stream = cfg.stream;
    return cudaSuccess;
}
static cudaError_t launch(int f, struct dim3 g, struct dim3 b, size_t smem)
{
    const int limit = fn[f].limit[device] ? fn[f].limit[device] : 48 * 1024;
    if (named(f, no_launch) || smem > (size_t)limit || !g.x || !g.y || !g.z || g.y > 65535 || g.z > 65535 || !b.x ||
        b.x * b.y * b.z > 1024) {
        ++fn[f].refused[device];
        return ret(cudaErrorInvalidValue);
    }
    ++fn[f].runs[device];
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *host) { *k = (cudaKernel_t)host; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, struct dim3 g, struct dim3 b, void **args, size_t smem, cudaStream_t s)
{
    (void)args; (void)s;
    return launch(find((const void *)k), g, b, smem);
}
cudaError_t cudaLaunchKernel(const void *f, struct dim3 g, struct dim3 b, void **args, size_t smem, cudaStream_t s)
{
    (void)args; (void)s;
    return launch(find(f), g, b, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args)
{
    (void)args;
    return launch(find(f), c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v)
{
    const int i = find(f);
    if (named(i, no_limit) || v > 227 * 1024) return ret(cudaErrorInvalidValue);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fn[i].limit[device] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *f, const cudaLaunchConfig_t *c)
{
    (void)c;
    if (named(find(f), no_cluster)) return ret(cudaErrorInvalidClusterSize);
    *n = clusters;
    return cudaSuccess;
}

/* devices and errors */
cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d)
{
    if (d < 0 || d > 1) return ret(cudaErrorInvalidDevice);
    device = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount       ? 152
         : a == cudaDevAttrComputeCapabilityMajor ? 10
         : a == cudaDevAttrComputeCapabilityMinor ? 3
                                                   : 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return last; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused by the test"; }

/* memory */
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = capacity - used; *t = capacity; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n)
{
    if (used + n > capacity) return ret(cudaErrorMemoryAllocation);
    if (n > largest) largest = n;
    for (int i = 0; i < MAXA; ++i)
        if (!mem[i].p) {
            *p = mmap(NULL, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
            if (*p == MAP_FAILED) abort();
            mem[i].p = *p;
            mem[i].bytes = n;
            used += n;
            return cudaSuccess;
        }
    abort();
}
cudaError_t cudaFree(void *p)
{
    for (int i = 0; p && i < MAXA; ++i)
        if (mem[i].p == p) { munmap(p, mem[i].bytes); mem[i].p = NULL; used -= mem[i].bytes; return cudaSuccess; }
    return p ? ret(cudaErrorInvalidValue) : cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) { (void)s; return cudaMemset(p, v, n); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)k; (void)st;
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *v, const void *s, size_t n, size_t o, enum cudaMemcpyKind k)
{
    (void)k;
    memcpy((char *)v + o, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void *d, const void *v, size_t n, size_t o, enum cudaMemcpyKind k)
{
    (void)k;
    memcpy(d, (const char *)v + o, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *v) { *p = (void *)v; return cudaSuccess; }

/* streams and events: nothing is asynchronous here */
static int handle;
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)&handle; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)&handle; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *t = 0; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
