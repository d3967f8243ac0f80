/* A CUDA runtime without a device, for tests of the library's host code: device
 * memory is host memory, copies copy, kernel launches are counted and do nothing.
 * Linked with the library's objects in place of the real runtime
 * (tests/fake_device.py).  A test can make allocations fail and can ask what was
 * launched, allocated and uploaded. */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAXL 65536
#define MAXF 4096

static const void *g_fun[MAXF];
static char *g_name[MAXF];
static int g_nfun;

static struct { const void *fun; dim3 grid, block; } g_launch[MAXL];
static int g_nlaunch;
static long g_mallocs, g_uploads, g_upload_bytes, g_live;
static int g_fail_after = -1, g_fail_count;
static char g_watch[64];
static int g_watch_arg = -1;
static unsigned char g_watched[128];

/* ---- what the tests call ---- */
void fake_clear(void) { g_nlaunch = 0; g_mallocs = g_uploads = g_upload_bytes = 0; }
/* the next `skip` allocations succeed, the `count` after them fail */
void fake_fail_malloc(int skip, int count) { g_fail_after = count > 0 ? skip : -1; g_fail_count = count; }
long fake_mallocs(void) { return g_mallocs; }
long fake_uploads(void) { return g_uploads; }
long fake_upload_bytes(void) { return g_upload_bytes; }
long fake_live_bytes(void) { return g_live; }
int fake_launches(void) { return g_nlaunch; }
const char *fake_launch(int k, unsigned *grid_block)
{
    int f;
    grid_block[0] = g_launch[k].grid.x; grid_block[1] = g_launch[k].grid.y; grid_block[2] = g_launch[k].grid.z;
    grid_block[3] = g_launch[k].block.x; grid_block[4] = g_launch[k].block.y; grid_block[5] = g_launch[k].block.z;
    for (f = 0; f < g_nfun; ++f)
        if (g_fun[f] == g_launch[k].fun) return g_name[f];
    return "";
}
/* remember the first 128 bytes of argument `arg` of kernels whose name holds `name` */
void fake_watch(const char *name, int arg)
{
    snprintf(g_watch, sizeof g_watch, "%s", name);
    g_watch_arg = arg;
    memset(g_watched, 0, sizeof g_watched);
}
void fake_watched(void *out) { memcpy(out, g_watched, sizeof g_watched); }

static cudaError_t launch(const void *fun, dim3 grid, dim3 block, void **args)
{
    int f;
    if (g_nlaunch < MAXL) {
        g_launch[g_nlaunch].fun = fun;
        g_launch[g_nlaunch].grid = grid;
        g_launch[g_nlaunch].block = block;
        ++g_nlaunch;
    }
    if (g_watch_arg >= 0)
        for (f = 0; f < g_nfun; ++f)
            if (g_fun[f] == fun && strstr(g_name[f], g_watch)) memcpy(g_watched, args[g_watch_arg], sizeof g_watched);
    return cudaSuccess;
}

/* ---- registration and launches ---- */
void **__cudaRegisterFatBinary(void *x) { (void)x; return (void **)calloc(1, sizeof(void *)); }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int tl, void *tid, void *bid,
                            dim3 *bd, dim3 *gd, int *ws)
{
    (void)h; (void)dev; (void)tl; (void)tid; (void)bid; (void)bd; (void)gd; (void)ws;
    if (g_nfun < MAXF) {
        g_fun[g_nfun] = host;
        g_name[g_nfun++] = strdup(name);
    }
}
void __cudaRegisterVar(void **h, char *hv, char *da, const char *dn, int e, size_t s, int c, int g)
{
    (void)h; (void)hv; (void)da; (void)dn; (void)e; (void)s; (void)c; (void)g;
}
char __cudaInitModule(void **h) { (void)h; return 1; }

static dim3 g_cg, g_cb;
static size_t g_cs;
static cudaStream_t g_cst;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st *st)
{
    g_cg = g; g_cb = b; g_cs = s; g_cst = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st)
{
    *g = g_cg; *b = g_cb; *s = g_cs; *(cudaStream_t *)st = g_cst;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t s, cudaStream_t st)
{
    (void)s; (void)st;
    return launch(f, g, b, a);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a)
{
    return launch(f, c->gridDim, c->blockDim, a);
}

/* ---- memory ---- */
cudaError_t cudaMalloc(void **p, size_t n)
{
    size_t *q;
    *p = NULL;
    if (g_fail_after == 0 && g_fail_count > 0) {
        if (--g_fail_count == 0) g_fail_after = -1;
        return cudaErrorMemoryAllocation;
    }
    if (g_fail_after > 0) --g_fail_after;
    if (posix_memalign((void **)&q, 512, n + 512)) return cudaErrorMemoryAllocation;
    memset(q, 0, n + 512);
    q[0] = n;
    *p = (char *)q + 512;
    ++g_mallocs;
    g_live += (long)n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (p) {
        g_live -= (long)*(size_t *)((char *)p - 512);
        free((char *)p - 512);
    }
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; *p = calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k)
{
    if (k == cudaMemcpyHostToDevice) {
        ++g_uploads;
        g_upload_bytes += (long)n;
    }
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemcpy2D(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k)
{
    size_t i;
    (void)k;
    for (i = 0; i < h; ++i) memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { (void)st; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)180 << 30; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { (void)s; *p = NULL; return cudaErrorInvalidSymbol; }

/* ---- device, streams, events, graphs ---- */
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int d)
{
    (void)d;
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl)
{
    (void)f; (void)b; (void)s; (void)fl;
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }

static int encode(void) { return 0; }   /* cuTensorMapEncodeTiled */
cudaError_t cudaGetDriverEntryPoint(const char *s, void **p, unsigned long long f, enum cudaDriverEntryPointQueryResult *q)
{
    (void)s; (void)f;
    *p = (void *)encode;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

static void *token(void) { return calloc(1, 8); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)token(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)token(); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)token(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = (cudaEvent_t)token(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned f) { (void)e; (void)s; (void)f; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *t = 0.001f; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) { (void)g; (void)f; *x = (cudaGraphExec_t)token(); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
