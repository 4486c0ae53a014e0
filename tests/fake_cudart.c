/* A CUDA runtime without a GPU, for tests of the library's host side.
 *
 * Device memory is host memory, copies are memcpy, kernels do not run.  What
 * the library asks of the runtime is kept: the bytes it allocates, and the
 * kernels it launches on a stream of its own while work on the legacy default
 * stream may still be under way.  As the runtime documents it, cudaMemset
 * returns before the memory is set, and cudaMemcpy from pageable memory waits
 * for the stream, stages the block and returns before the transfer has ended;
 * a non-blocking stream is not ordered after either.
 */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef struct { unsigned x, y, z; } dim3_t;

static int pending;                 /* the legacy stream may be busy */
static int launches, violations;
static char first_violation[256];
static size_t allocated, malloc_limit = (size_t)-1;
static int pinned;                  /* what cudaPointerGetAttributes says */

static struct { const char *name; unsigned block; } last[512];   /* each kernel's last block size */
static int nlast;
unsigned fake_block_of(const char *part)
{
    for (int i = 0; i < nlast; ++i)
        if (strstr(last[i].name, part)) return last[i].block;
    return 0;
}

void fake_reset(void) { launches = violations = 0; first_violation[0] = 0; allocated = 0; malloc_limit = (size_t)-1; pinned = 0; nlast = 0; }
int fake_launches(void) { return launches; }
int fake_violations(void) { return violations; }
const char *fake_first_violation(void) { return first_violation; }
size_t fake_allocated(void) { return allocated; }
void fake_malloc_limit(size_t bytes) { malloc_limit = bytes; }
void fake_pinned(int on) { pinned = on; }

/* ---- registration and launches ---- */
static struct { const void *host; const char *name; } kernels[4096];
static int nkernels;
static int handle;

void **__cudaRegisterFatBinary(void *fat) { static void *h; (void)fat; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *a, char *b, const char *c, int e, size_t s, int k, int g)
{ (void)h, (void)a, (void)b, (void)c, (void)e, (void)s, (void)k, (void)g; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int lim, void *t, void *b,
                            void *bd, void *gd, int *ws)
{
    (void)h, (void)dev, (void)lim, (void)t, (void)b, (void)bd, (void)gd, (void)ws;
    if (nkernels < 4096) kernels[nkernels].host = host, kernels[nkernels++].name = name;
}
static struct { dim3_t g, b; size_t smem; void *stream; } cfg;
unsigned __cudaPushCallConfiguration(dim3_t g, dim3_t b, size_t smem, void *stream)
{ cfg.g = g, cfg.b = b, cfg.smem = smem, cfg.stream = stream; return 0; }
err_t __cudaPopCallConfiguration(dim3_t *g, dim3_t *b, size_t *smem, void *stream)
{ *g = cfg.g, *b = cfg.b, *smem = cfg.smem, *(void **)stream = cfg.stream; return 0; }
err_t __cudaGetKernel(void **k, const void *host)
{
    for (int i = 0; i < nkernels; ++i)
        if (kernels[i].host == host) { *k = (void *)kernels[i].name; return 0; }
    *k = (void *)"?";
    return 0;
}
err_t __cudaLaunchKernel(void *k, dim3_t g, dim3_t b, void **args, size_t smem, void *stream)
{
    (void)args, (void)smem;
    ++launches;
    if (g.x == 0 || b.x == 0 || b.x > 1024) return 9;   /* cudaErrorInvalidConfiguration */
    int i = 0;
    while (i < nlast && last[i].name != (char *)k) ++i;
    if (i < 512) last[i].name = k, last[i].block = b.x, nlast += i == nlast;
    if (stream && pending && violations++ == 0) snprintf(first_violation, sizeof first_violation, "%s", (char *)k);
    return 0;
}

/* ---- memory ---- */
err_t cudaMalloc(void **p, size_t n)
{
    if (n > malloc_limit || !(*p = calloc(n ? n : 1, 1))) return 2;   /* cudaErrorMemoryAllocation */
    allocated += n;
    return 0;
}
err_t cudaFree(void *p) { free(p); return 0; }
err_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)1 << 40; return 0; }
err_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); pending = 1; return 0; }
err_t cudaMemsetAsync(void *p, int v, size_t n, void *s) { (void)s; memset(p, v, n); return 0; }
err_t cudaMemcpy(void *d, const void *s, size_t n, int kind) { memcpy(d, s, n); pending = kind == 1; return 0; }
err_t cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) { (void)kind, (void)st; memcpy(d, s, n); return 0; }
err_t cudaGetSymbolAddress(void **p, const void *s) { *p = (void *)s; return 0; }
err_t cudaPointerGetAttributes(void *a, const void *p) { (void)p; memset(a, 0, 16); *(int *)a = pinned; return 0; }

/* ---- streams, events, graphs ---- */
err_t cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; *s = &handle; return 0; }
err_t cudaStreamDestroy(void *s) { (void)s; return 0; }
err_t cudaStreamSynchronize(void *s) { if (!s) pending = 0; return 0; }
err_t cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)s, (void)e, (void)f; return 0; }
err_t cudaStreamIsCapturing(void *s, int *c) { (void)s; *c = 0; return 0; }
err_t cudaStreamBeginCapture(void *s, int m) { (void)s, (void)m; return 0; }
err_t cudaStreamEndCapture(void *s, void **g) { (void)s; *g = &handle; return 0; }
err_t cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; *e = &handle; return 0; }
err_t cudaEventDestroy(void *e) { (void)e; return 0; }
err_t cudaEventRecord(void *e, void *s) { (void)e, (void)s; return 0; }
err_t cudaEventRecordWithFlags(void *e, void *s, unsigned f) { (void)e, (void)s, (void)f; return 0; }
err_t cudaGraphInstantiate(void **x, void *g, unsigned long long f) { (void)g, (void)f; *x = &handle; return 0; }
err_t cudaGraphLaunch(void *x, void *s) { (void)x, (void)s; return 0; }
err_t cudaGraphDestroy(void *g) { (void)g; return 0; }
err_t cudaGraphExecDestroy(void *x) { (void)x; return 0; }
err_t cudaGetDevice(int *d) { *d = 0; return 0; }
err_t cudaGetLastError(void) { return 0; }
err_t cudaPeekAtLastError(void) { return 0; }
const char *cudaGetErrorString(err_t e) { return e == 2 ? "out of memory" : "error"; }
