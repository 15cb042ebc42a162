/* A CUDA runtime without a device: device memory is host memory, kernels are
 * counted and not run.  Linked with the library's own objects, it shows what
 * the host code does when an allocation fails, and what it leaves behind. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

enum { OK = cudaSuccess, INVALID = cudaErrorInvalidValue, NO_MEMORY = cudaErrorMemoryAllocation, BAD_GRID = cudaErrorInvalidConfiguration };
enum { SLOTS = 4096 };
static struct { char* p; size_t n; } g_mem[SLOTS];
static cudaError_t g_last;
static int g_countdown = -1, g_launches;
static size_t g_capacity = (size_t)1 << 32, g_used;

/* What a test sets and reads. */
void fake_reset(void) { g_last = OK; g_countdown = -1; g_launches = 0; g_capacity = (size_t)1 << 32; }
void fake_fail_after(int n) { g_countdown = n; } /* the n-th allocation from now on (from 0) fails, once */
int fake_pending(void) { return g_countdown >= 0; }
void fake_set_capacity(size_t n) { g_capacity = n; }
int fake_launches(void) { return g_launches; }
size_t fake_used(void) { return g_used; }
int fake_holds(const void* bytes, size_t n) { /* whether live device memory holds these bytes */
    for (int i = 0; i < SLOTS; i++)
        if (g_mem[i].p && memmem(g_mem[i].p, g_mem[i].n, bytes, n)) return 1;
    return 0;
}

static cudaError_t done(cudaError_t e) {
    if (e) g_last = e;
    return e;
}
static cudaError_t get(void** out, size_t n) {
    if (g_countdown >= 0 && g_countdown-- == 0) return done(NO_MEMORY);
    if (g_used + n > g_capacity) return done(NO_MEMORY);
    for (int i = 0; i < SLOTS; i++)
        if (!g_mem[i].p) {
            if (!(g_mem[i].p = calloc(1, n ? n : 1))) return done(NO_MEMORY);
            g_mem[i].n = n;
            g_used += n;
            *out = g_mem[i].p;
            return OK;
        }
    return done(NO_MEMORY);
}
static cudaError_t put(void* p) {
    if (!p) return OK;
    for (int i = 0; i < SLOTS; i++)
        if (g_mem[i].p == p) {
            g_used -= g_mem[i].n;
            free(p);
            g_mem[i].p = 0;
            return OK;
        }
    return done(INVALID);
}

cudaError_t cudaMalloc(void** p, size_t n) { return get(p, n); }
cudaError_t cudaFree(void* p) { return put(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return get(p, n); }
cudaError_t cudaFreeHost(void* p) { return put(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { (void)k; memcpy(d, s, n); return OK; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)k; (void)st;
    memcpy(d, s, n);
    return OK;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { (void)st; memset(d, v, n); return OK; }
cudaError_t cudaMemcpyToSymbolAsync(const void* y, const void* s, size_t n, size_t o, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)y; (void)s; (void)n; (void)o; (void)k; (void)st;
    return OK;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* y) { *p = (void*)y; return OK; }
cudaError_t cudaGetLastError(void) { cudaError_t e = g_last; g_last = OK; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == NO_MEMORY ? "out of memory" : "an error"; }

cudaError_t cudaGetDevice(int* d) { *d = 0; return OK; }
cudaError_t cudaSetDevice(int d) { return done(d ? INVALID : OK); }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return OK; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int d) { /* a B200's, as far as the library asks */
    (void)d;
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return OK;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { (void)a; (void)d; *v = 148; return OK; }
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void* f) { (void)a; (void)f; return done(INVALID); }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return OK; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* s, void** f, unsigned v, unsigned long long g,
                                             enum cudaDriverEntryPointQueryResult* q) {
    (void)s; (void)v; (void)g; (void)q;
    *f = 0;
    return done(INVALID);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int t, size_t s) {
    (void)f; (void)s;
    *n = 512 / t;
    return OK;
}

/* Streams, events and graphs are allocations too: a lost one shows. */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { (void)f; return get((void**)s, 1); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return put(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return OK; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return OK; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) { (void)s; return get((void**)g, 1); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long f) { (void)g; (void)f; return get((void**)e, 1); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { (void)e; (void)s; g_launches++; return OK; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return put(g); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return put(e); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return get((void**)e, 1); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return put(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return OK; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return OK; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 1.0f; return OK; }

/* What nvcc's launch syntax and its kernel registration call. */
static struct { dim3 g, b; size_t s; void* st; } g_conf;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
    g_conf.g = g;
    g_conf.b = b;
    g_conf.s = s;
    g_conf.st = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    *g = g_conf.g;
    *b = g_conf.b;
    *s = g_conf.s;
    *(void**)st = g_conf.st;
    return OK;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st) {
    (void)f; (void)b; (void)a; (void)s; (void)st;
    if (!g.x) return done(BAD_GRID);
    g_launches++;
    return OK;
}
void** __cudaRegisterFatBinary(void* f) { static void* h; (void)f; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* n, int l, void* t, void* i, void* b, void* g, int* w) {
    (void)h; (void)f; (void)d; (void)n; (void)l; (void)t; (void)i; (void)b; (void)g; (void)w;
}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {
    (void)h; (void)v; (void)d; (void)n; (void)e; (void)s; (void)c; (void)g;
}
