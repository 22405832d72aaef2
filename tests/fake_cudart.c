/* A stand-in for the CUDA runtime, for host-side tests without a GPU: device memory is zeroed host memory, kernels do
 * nothing, streams run in order at once. It counts what the library holds and logs what it asks for, pretends to have
 * several devices, and fails a chosen kernel's launch. Built and loaded under the runtime's name by
 * tests/test_host_resources_cpu.py. Signatures are those of the public runtime API and of nvcc's host stubs. */
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;
typedef struct { unsigned x, y, z; } dim3_t;
enum { OK = 0, LAUNCH_FAILURE = 719 };

/* what the tests steer and read */
static int g_device, g_devices = 2;
static unsigned long long g_context[64];
static long g_host_blocks, g_streams, g_events, g_device_blocks;
static char g_fail[128];
static unsigned char g_patch[4096];
static size_t g_patch_at, g_patch_len;
static char *g_log;
static size_t g_log_len, g_log_cap;

void fake_set_device(int d) { g_device = d; }
void fake_new_context(int d) { g_context[d] += 64; }
long fake_host_blocks(void) { return g_host_blocks; }
long fake_streams(void) { return g_streams; }
long fake_events(void) { return g_events; }
long fake_device_blocks(void) { return g_device_blocks; }
void fake_fail_launch(const char *kernel) { snprintf(g_fail, sizeof(g_fail), "%s", kernel); }
/* the next device-to-host copies of exactly `size` bytes start with the len bytes at p */
void fake_patch(size_t size, const void *p, size_t len) {
    g_patch_at = size;
    g_patch_len = len;
    memcpy(g_patch, p, len);
}
const char *fake_log(void) { return g_log ? g_log : ""; }
void fake_clear_log(void) {
    g_log_len = 0;
    if (g_log) g_log[0] = 0;
}
static void note(const char *what, const void *a, const void *b) {
    char line[256];
    const int n = snprintf(line, sizeof(line), "%s %p %p\n", what, a, b);
    if (g_log_len + n + 1 > g_log_cap) {
        g_log_cap = 2 * g_log_cap + 4096;
        g_log = realloc(g_log, g_log_cap);
    }
    memcpy(g_log + g_log_len, line, n + 1);
    g_log_len += n;
}

/* kernels */
typedef struct { const void *host; const char *name; } kernel_t;
static kernel_t g_kernels[4096];
static int g_nkernels;
static const char *name_of(const void *f) {
    for (int i = 0; i < g_nkernels; i++)
        if (g_kernels[i].host == f) return g_kernels[i].name;
    return "unknown";
}
static err_t launched(const void *f, void *stream) {
    const char *name = name_of(f);
    char what[200];
    if (g_fail[0] && strstr(name, g_fail)) {
        g_fail[0] = 0;
        note("failed-launch", NULL, stream);
        return LAUNCH_FAILURE;
    }
    snprintf(what, sizeof(what), "launch:%s", name);
    note(what, NULL, stream);
    return OK;
}
void **__cudaRegisterFatBinary(void *b) {
    static void *handle;
    handle = b;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int lim, void *t, void *b, void *bd,
                            void *gd, int *w) {
    (void)h, (void)dev, (void)lim, (void)t, (void)b, (void)bd, (void)gd, (void)w;
    if (g_nkernels < 4096) g_kernels[g_nkernels++] = (kernel_t){host, name};
}
void __cudaRegisterVar(void **h, char *host, char *dev, const char *name, int ext, size_t size, int c, int g) {
    (void)h, (void)host, (void)dev, (void)name, (void)ext, (void)size, (void)c, (void)g;
}
err_t __cudaGetKernel(void **k, const void *f) {
    *k = (void *)f;
    return OK;
}
static struct { dim3_t grid, block; size_t smem; void *stream; } g_call;
unsigned __cudaPushCallConfiguration(dim3_t grid, dim3_t block, size_t smem, void *stream) {
    g_call.grid = grid, g_call.block = block, g_call.smem = smem, g_call.stream = stream;
    return 0;
}
err_t __cudaPopCallConfiguration(dim3_t *grid, dim3_t *block, size_t *smem, void *stream) {
    *grid = g_call.grid, *block = g_call.block, *smem = g_call.smem, *(void **)stream = g_call.stream;
    return OK;
}
err_t __cudaLaunchKernel(void *k, dim3_t grid, dim3_t block, void **args, size_t smem, void *stream) {
    (void)grid, (void)block, (void)args, (void)smem;
    return launched(k, stream);
}
err_t cudaLaunchKernel(const void *f, dim3_t grid, dim3_t block, void **args, size_t smem, void *stream) {
    (void)grid, (void)block, (void)args, (void)smem;
    return launched(f, stream);
}
typedef struct { dim3_t grid, block; size_t smem; void *stream; } config_t;  /* cudaLaunchConfig_t's first members */
err_t cudaLaunchKernelExC(const config_t *c, const void *f, void **args) {
    (void)args;
    return launched(f, c->stream);
}

/* devices and contexts */
err_t cudaGetDevice(int *d) { *d = g_device; return OK; }
err_t cudaGetDeviceCount(int *n) { *n = g_devices; return OK; }
err_t cudaDeviceGetAttribute(int *v, int a, int d) { (void)a, (void)d; *v = 8; return OK; }
static int ctx_get_current(void **c) { *c = &g_context[g_device]; return 0; }
static int ctx_get_id(void *c, unsigned long long *id) {
    *id = *(unsigned long long *)c + (unsigned long long)((unsigned long long *)c - g_context) + 1;
    return 0;
}
err_t cudaGetDriverEntryPointByVersion(const char *s, void **p, unsigned v, unsigned long long f, int *found) {
    (void)v, (void)f;
    *p = !strcmp(s, "cuCtxGetCurrent") ? (void *)ctx_get_current : !strcmp(s, "cuCtxGetId") ? (void *)ctx_get_id : NULL;
    if (found) *found = *p ? 0 : 1;
    return *p ? OK : 500;
}
err_t cudaDeviceSynchronize(void) { return OK; }
err_t cudaGetLastError(void) { return OK; }
const char *cudaGetErrorString(err_t e) { return e ? "failure made by the test" : "no error"; }

/* memory */
static void *device_block(size_t n) {
    g_device_blocks++;
    return calloc(1, n ? n : 1);
}
err_t cudaMalloc(void **p, size_t n) { *p = device_block(n); return OK; }
err_t cudaFree(void *p) { if (p) g_device_blocks--; free(p); return OK; }
err_t cudaMallocAsync(void **p, size_t n, void *s) { (void)s; return cudaMalloc(p, n); }
err_t cudaMallocFromPoolAsync(void **p, size_t n, void *pool, void *s) { (void)pool, (void)s; return cudaMalloc(p, n); }
err_t cudaFreeAsync(void *p, void *s) {
    note("free", p, s);
    return cudaFree(p);
}
err_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; *p = calloc(1, n); g_host_blocks++; return OK; }
err_t cudaFreeHost(void *p) { free(p); g_host_blocks--; return OK; }
err_t cudaMemGetInfo(size_t *a, size_t *b) { *a = *b = (size_t)1 << 34; return OK; }
err_t cudaMemPoolCreate(void **p, const void *props) { (void)props; *p = malloc(1); return OK; }
err_t cudaMemPoolSetAttribute(void *p, int a, void *v) { (void)p, (void)a, (void)v; return OK; }
err_t cudaMemPoolGetAttribute(void *p, int a, void *v) { (void)p, (void)a; memset(v, 0, 8); return OK; }
err_t cudaMemcpy(void *d, const void *s, size_t n, int k) {
    memmove(d, s, n);
    if (k == 2 && n == g_patch_at && g_patch_len) memcpy(d, g_patch, g_patch_len);
    return OK;
}
err_t cudaMemcpyAsync(void *d, const void *s, size_t n, int k, void *st) { (void)st; return cudaMemcpy(d, s, n, k); }
err_t cudaMemsetAsync(void *d, int v, size_t n, void *st) { (void)st; memset(d, v, n); return OK; }
err_t cudaPointerGetAttributes(void *a, const void *p) { (void)p; memset(a, 0, 32); return OK; }
err_t cudaGetSymbolAddress(void **p, const void *s) { *p = (void *)s; return OK; }
err_t cudaFuncSetAttribute(const void *f, int a, int v) { (void)f, (void)a, (void)v; return OK; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
    (void)f, (void)b, (void)s, (void)fl;
    *n = 1;
    return OK;
}

/* streams and events: their device, which cudaStreamGetDevice gives back */
err_t cudaStreamCreateWithFlags(void **s, unsigned f) {
    (void)f;
    int *d = malloc(sizeof(int));
    *d = g_device;
    *s = d;
    g_streams++;
    return OK;
}
err_t cudaStreamDestroy(void *s) { free(s); g_streams--; return OK; }
err_t cudaStreamGetDevice(void *s, int *d) { *d = s ? *(int *)s : g_device; return OK; }
err_t cudaStreamSynchronize(void *s) { note("synchronize", NULL, s); return OK; }
err_t cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)f; note("wait", e, s); return OK; }
err_t cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; *e = malloc(1); g_events++; return OK; }
err_t cudaEventCreate(void **e) { return cudaEventCreateWithFlags(e, 0); }
err_t cudaEventDestroy(void *e) { free(e); g_events--; return OK; }
err_t cudaEventRecord(void *e, void *s) { note("record", e, s); return OK; }
err_t cudaEventSynchronize(void *e) { (void)e; return OK; }
err_t cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a, (void)b; *ms = 0.f; return OK; }

/* graphs: nothing is captured, a launch is logged */
err_t cudaStreamBeginCapture(void *s, int m) { (void)s, (void)m; return OK; }
err_t cudaStreamEndCapture(void *s, void **g) { (void)s; *g = malloc(1); return OK; }
err_t cudaGraphInstantiate(void **e, void *g, unsigned long long f) { (void)g, (void)f; *e = malloc(1); return OK; }
err_t cudaGraphGetNodes(void *g, void **n, size_t *k) { (void)g, (void)n; *k = 0; return OK; }
err_t cudaGraphNodeGetType(void *n, int *t) { (void)n; *t = 0; return OK; }
err_t cudaGraphLaunch(void *e, void *s) { note("graph-launch", e, s); return OK; }
err_t cudaGraphExecDestroy(void *e) { free(e); return OK; }
err_t cudaGraphDestroy(void *g) { free(g); return OK; }
