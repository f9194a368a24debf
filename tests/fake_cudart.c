/* A CUDA runtime without a GPU, preloaded under liblux_gpu.so to test its host code: device
 * memory is host memory within a limit, copies and memsets are done at once, kernels are
 * recorded and not run.  The record is text, one call a line (fake_log). */
#define _GNU_SOURCE
#include <pthread.h>
#include <stdarg.h>
#include <stddef.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

typedef int err_t;                       /* cudaError_t */
enum { kOk = 0, kInvalid = 1, kMemory = 2 };
typedef struct { unsigned x, y, z; } dim3_t;

static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static char *log_text;
static size_t log_len, log_cap;
static size_t limit_bytes = (size_t)1 << 33, used_bytes;
static struct { char *p; size_t bytes; } blocks[4096];
static int block_count;
static struct { const void *host; const char *name; } kernels[1024];
static int kernel_count;

static void say(const char *fmt, ...) {
    char line[512];
    va_list ap;
    va_start(ap, fmt);
    int n = vsnprintf(line, sizeof line, fmt, ap);
    va_end(ap);
    pthread_mutex_lock(&mu);
    if (log_len + n + 2 > log_cap) {
        log_cap = 2 * log_cap + 4096;
        log_text = realloc(log_text, log_cap);
    }
    memcpy(log_text + log_len, line, n);
    log_len += n;
    log_text[log_len++] = '\n';
    log_text[log_len] = 0;
    pthread_mutex_unlock(&mu);
}

const char *fake_log(void) { return log_text ? log_text : ""; }
void fake_clear_log(void) { if (log_text) log_text[log_len = 0] = 0; }
void fake_set_limit(size_t bytes) { limit_bytes = bytes; }
size_t fake_used(void) { return used_bytes; }

static err_t take(void **p, size_t bytes) {
    *p = NULL;
    pthread_mutex_lock(&mu);
    err_t err = kMemory;
    if (used_bytes + bytes <= limit_bytes && block_count < 4096) {
        char *m = calloc(bytes ? bytes : 1, 1);
        blocks[block_count].p = m;
        blocks[block_count++].bytes = bytes;
        used_bytes += bytes;
        *p = m;
        err = kOk;
    }
    pthread_mutex_unlock(&mu);
    say("malloc %zu %p", bytes, *p);
    return err;
}
static err_t give(void *p) {
    if (!p) return kOk;
    pthread_mutex_lock(&mu);
    err_t err = kInvalid;
    for (int i = 0; i < block_count; ++i)
        if (blocks[i].p == p) {
            used_bytes -= blocks[i].bytes;
            free(p);
            blocks[i] = blocks[--block_count];
            err = kOk;
            break;
        }
    pthread_mutex_unlock(&mu);
    if (err) say("free of an unknown pointer");
    return err;
}
static int on_device(const void *p) {
    int found = 0;
    pthread_mutex_lock(&mu);
    for (int i = 0; i < block_count && !found; ++i)
        found = (const char *)p >= blocks[i].p && (const char *)p < blocks[i].p + blocks[i].bytes;
    pthread_mutex_unlock(&mu);
    return found;
}

/* ---- registration and launches */
void **__cudaRegisterFatBinary(void *f) { static void *h; (void)f; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *hv, char *da, const char *dn, int e, size_t s, int c, int g) {
    (void)h; (void)hv; (void)da; (void)dn; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int limit,
                            void *tid, void *bid, void *bdim, void *gdim, int *ws) {
    (void)h; (void)dev; (void)limit; (void)tid; (void)bid; (void)bdim; (void)gdim; (void)ws;
    if (kernel_count < 1024) {
        kernels[kernel_count].host = host;
        kernels[kernel_count++].name = name;
    }
}
static __thread struct { dim3_t grid, block; size_t smem; void *stream; } pending;
unsigned __cudaPushCallConfiguration(dim3_t grid, dim3_t block, size_t smem, void *stream) {
    pending.grid = grid; pending.block = block; pending.smem = smem; pending.stream = stream;
    return 0;
}
err_t __cudaPopCallConfiguration(dim3_t *grid, dim3_t *block, size_t *smem, void *stream) {
    *grid = pending.grid; *block = pending.block; *smem = pending.smem;
    *(void **)stream = pending.stream;
    return kOk;
}
err_t cudaLaunchKernel(const void *fn, dim3_t grid, dim3_t block, void **args, size_t smem,
                       void *stream) {
    const char *name = "?";
    for (int i = 0; i < kernel_count; ++i) if (kernels[i].host == fn) name = kernels[i].name;
    (void)block; (void)args; (void)smem;
    say("launch %s grid %u stream %p", name, grid.x, stream);
    return kOk;
}

/* ---- memory */
err_t cudaMalloc(void **p, size_t bytes) { return take(p, bytes); }
err_t cudaFree(void *p) { return give(p); }
err_t cudaMallocHost(void **p, size_t bytes) { return (*p = calloc(bytes ? bytes : 1, 1)) ? kOk : kMemory; }
err_t cudaFreeHost(void *p) { free(p); return kOk; }
err_t cudaMallocFromPoolAsync(void **p, size_t bytes, void *pool, void *s) { (void)pool; (void)s; return take(p, bytes); }
err_t cudaFreeAsync(void *p, void *s) { (void)s; return give(p); }
err_t cudaMemcpy(void *d, const void *s, size_t n, int kind) {
    (void)kind; say("memcpy %zu stream default", n); memcpy(d, s, n); return kOk;
}
err_t cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st) {
    (void)kind; say("memcpy %zu stream %p", n, st); memcpy(d, s, n); return kOk;
}
err_t cudaMemset(void *p, int v, size_t n) {
    say("memset %zu stream default", n); memset(p, v, n); return kOk;
}
err_t cudaMemsetAsync(void *p, int v, size_t n, void *st) {
    say("memset %zu stream %p", n, st); memset(p, v, n); return kOk;
}
struct attributes { int type, device; void *device_pointer, *host_pointer; };
err_t cudaPointerGetAttributes(struct attributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    a->type = on_device(p) ? 2 : 0;
    return kOk;
}
err_t cudaGetSymbolAddress(void **p, const void *s) { (void)p; (void)s; return kInvalid; }

/* ---- devices, streams, events, graphs */
err_t cudaGetDeviceCount(int *n) { *n = 1; return kOk; }
err_t cudaSetDevice(int d) { (void)d; return kOk; }
err_t cudaDeviceGetAttribute(int *v, int a, int d) { (void)a; (void)d; *v = 148; return kOk; }
err_t cudaDeviceSynchronize(void) { return kOk; }
err_t cudaGetLastError(void) { return kOk; }
const char *cudaGetErrorString(err_t e) { return e == kMemory ? "out of memory" : e ? "error" : "no error"; }
err_t cudaFuncSetAttribute(const void *f, int a, int v) { (void)f; (void)a; (void)v; return kOk; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned g) {
    (void)f; (void)b; (void)s; (void)g; *n = 4; return kOk;
}
static err_t handle(void **p) { *p = calloc(1, 8); return kOk; }
static err_t drop(void *p) { free(p); return kOk; }
err_t cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; return handle(s); }
err_t cudaStreamDestroy(void *s) { return drop(s); }
err_t cudaStreamSynchronize(void *s) { (void)s; return kOk; }
err_t cudaStreamWaitEvent(void *s, void *e, unsigned f) { (void)s; (void)e; (void)f; return kOk; }
err_t cudaStreamBeginCapture(void *s, int m) { (void)s; (void)m; return kOk; }
err_t cudaStreamEndCapture(void *s, void **g) { (void)s; return handle(g); }
err_t cudaGraphInstantiate(void **e, void *g, unsigned long long f) { (void)g; (void)f; return handle(e); }
err_t cudaGraphLaunch(void *e, void *s) { (void)e; say("graph stream %p", s); return kOk; }
err_t cudaGraphDestroy(void *g) { return drop(g); }
err_t cudaGraphExecDestroy(void *e) { return drop(e); }
err_t cudaEventCreate(void **e) { return handle(e); }
err_t cudaEventCreateWithFlags(void **e, unsigned f) { (void)f; return handle(e); }
err_t cudaEventDestroy(void *e) { return drop(e); }
err_t cudaEventRecord(void *e, void *s) { (void)e; (void)s; return kOk; }
err_t cudaEventQuery(void *e) { (void)e; return kOk; }
err_t cudaEventSynchronize(void *e) { (void)e; return kOk; }
err_t cudaEventElapsedTime(float *ms, void *a, void *b) { (void)a; (void)b; *ms = 1.0f; return kOk; }
err_t cudaMemPoolCreate(void **p, const void *props) { (void)props; return handle(p); }
err_t cudaMemPoolDestroy(void *p) { return drop(p); }
err_t cudaMemPoolSetAttribute(void *p, int a, void *v) { (void)p; (void)a; (void)v; return kOk; }
