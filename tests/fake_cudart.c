/*
 * The CUDA runtime calls of libgame_gb300.so on host memory, for tests that
 * need a failing allocation or an account of the device memory and have no
 * GPU: device memory is calloc'd, copies are memcpy, kernels are counted and
 * not run.  Preloaded in front of libcudart (fakecuda.py).
 */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef struct {
    unsigned x, y, z;
} dim;
enum { MEMORY_ALLOCATION = 2 };

static long g_mallocs, g_fail_at = -1, g_launches;
static size_t g_live;
static err_t g_last;
static int g_streams;
static int g_handles;
static long g_unordered; /* clears on the default stream once other streams exist */

/* the n-th allocation from now (0 the next) fails, and every one after it
 * while keep is set; n < 0: none */
static int g_keep;
void fake_fail_malloc(long n, int keep)
{
    g_fail_at = n < 0 ? -1 : g_mallocs + n;
    g_keep = keep;
}
long fake_mallocs(void) { return g_mallocs; }
long fake_launches(void) { return g_launches; }
long fake_unordered_clears(void) { return g_unordered; }
size_t fake_live_bytes(void) { return g_live; }

err_t cudaMalloc(void **p, size_t n)
{
    const long k = g_mallocs++;
    if (g_fail_at >= 0 && (k == g_fail_at || (g_keep && k > g_fail_at))) return g_last = MEMORY_ALLOCATION;
    size_t *h = calloc(1, n + 64);
    if (!h) return g_last = MEMORY_ALLOCATION;
    *h = n;
    g_live += n;
    *p = (char *)h + 64;
    return 0;
}
err_t cudaFree(void *p)
{
    if (!p) return 0;
    size_t *h = (size_t *)((char *)p - 64);
    g_live -= *h;
    free(h);
    return 0;
}
err_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; return (*p = calloc(1, n)) ? 0 : (g_last = MEMORY_ALLOCATION); }
err_t cudaFreeHost(void *p) { free(p); return 0; }
err_t cudaHostGetDevicePointer(void **d, void *h, unsigned f) { (void)f; *d = h; return 0; }
err_t cudaMemcpy(void *d, const void *s, size_t n, int kind) { (void)kind; memmove(d, s, n); return 0; }
err_t cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) { (void)kind; (void)st; memmove(d, s, n); return 0; }
err_t cudaMemsetAsync(void *d, int v, size_t n, void *st) { g_unordered += !st && g_streams > 0; memset(d, v, n); return 0; }
err_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, 0); }
err_t cudaGetLastError(void) { err_t e = g_last; g_last = 0; return e; }
const char *cudaGetErrorString(err_t e) { return e == MEMORY_ALLOCATION ? "out of memory" : e ? "error" : "no error"; }
err_t cudaDeviceSynchronize(void) { return 0; }
err_t cudaGetDevice(int *d) { *d = 0; return 0; }
err_t cudaSetDevice(int d) { (void)d; return 0; }
err_t cudaGetSymbolAddress(void **p, const void *s) { (void)s; (void)p; return g_last = 13; }
static err_t handle(void **h) { *h = (void *)(size_t)(++g_handles); return 0; }
err_t cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; ++g_streams; return handle(s); }
err_t cudaStreamDestroy(void *s) { (void)s; --g_streams; return 0; }
err_t cudaStreamSynchronize(void *s) { (void)s; return 0; }
err_t cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)s; (void)e; (void)f; return 0; }
err_t cudaStreamIsCapturing(void *s, int *c) { (void)s; *c = 0; return 0; }
err_t cudaStreamBeginCapture(void *s, int m) { (void)s; (void)m; return 0; }
err_t cudaStreamEndCapture(void *s, void **g) { (void)s; return handle(g); }
err_t cudaGraphInstantiate(void **x, void *g, unsigned long long f) { (void)g; (void)f; return handle(x); }
err_t cudaGraphLaunch(void *x, void *s) { (void)x; (void)s; return 0; }
err_t cudaGraphDestroy(void *g) { (void)g; return 0; }
err_t cudaGraphExecDestroy(void *x) { (void)x; return 0; }
err_t cudaEventCreate(void **e) { return handle(e); }
err_t cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; return handle(e); }
err_t cudaEventDestroy(void *e) { (void)e; return 0; }
err_t cudaEventRecord(void *e, void *s) { (void)e; (void)s; return 0; }
err_t cudaEventRecordWithFlags(void *e, void *s, unsigned f) { (void)e; (void)s; (void)f; return 0; }
err_t cudaEventSynchronize(void *e) { (void)e; return 0; }
err_t cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 0.f; return 0; }

static dim g_grid, g_block;
static size_t g_smem;
static void *g_stream;
unsigned __cudaPushCallConfiguration(dim g, dim b, size_t m, void *s) { g_grid = g; g_block = b; g_smem = m; g_stream = s; return 0; }
err_t __cudaPopCallConfiguration(dim *g, dim *b, size_t *m, void *s) { *g = g_grid; *b = g_block; *m = g_smem; *(void **)s = g_stream; return 0; }
err_t __cudaGetKernel(void **k, const void *f) { *k = (void *)f; return 0; }
err_t __cudaLaunchKernel(void *k, dim g, dim b, void **a, size_t m, void *s)
{
    (void)k; (void)g; (void)b; (void)a; (void)m; (void)s;
    ++g_launches;
    return 0;
}
void **__cudaRegisterFatBinary(void *f) { (void)f; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *n, int t, void *a, void *b, void *c, void *e, int *w)
{
    (void)h; (void)f; (void)d; (void)n; (void)t; (void)a; (void)b; (void)c; (void)e; (void)w;
}
void __cudaRegisterVar(void **h, char *v, char *d, const char *n, int e, size_t s, int c, int g)
{
    (void)h; (void)v; (void)d; (void)n; (void)e; (void)s; (void)c; (void)g;
}
