/* A stand-in for the CUDA runtime, preloaded before the library in a child process: the host side of the
 * library (allocations, dispatch, launch set-up) runs on a machine without a GPU. Memory is host memory, kernels
 * are recorded by name and not run, and any call can be told to fail. Two devices. As on a GPU, a launch with
 * more than 48 KB of dynamic shared memory fails unless its kernel was given that much on the current device. */
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define NFUN 4096
#define NMEM 4096

static int device_now;
static cudaError_t last_error;
static struct { const void *host; char name[512]; int smem[2]; } fun[NFUN];
static int nfun;
static struct { char *p; size_t bytes; int type; } mem[NMEM];
static char *log_text;
static size_t log_len, log_cap;
static char fail_name[64];
static int fail_after;
static struct { dim3 grid, block; size_t smem; cudaStream_t s; } call[16];
static int ncall;

static void note(const char *what, const char *name, long n) {
    char line[640];
    const size_t k = (size_t)snprintf(line, sizeof line, "%s %s %ld\n", what, name, n);
    if (log_len + k + 1 > log_cap) log_text = realloc(log_text, log_cap = 2 * log_cap + k + 4096);
    memcpy(log_text + log_len, line, k + 1);
    log_len += k;
}

const char *fake_log(void) { return log_text ? log_text : ""; }
void fake_reset(void) { log_len = 0; if (log_text) log_text[0] = 0; }
/* the nth call from now of the function fails with cudaErrorMemoryAllocation */
void fake_fail(const char *name, int nth) { snprintf(fail_name, sizeof fail_name, "%s", name); fail_after = nth; }
long fake_live(void) { long n = 0; for (int i = 0; i < NMEM; i++) n += mem[i].p != NULL; return n; }

static int failing(const char *name) { return fail_after && !strcmp(name, fail_name) && --fail_after == 0; }
static cudaError_t set(cudaError_t e) { if (e) last_error = e; return e; }

static cudaError_t get_memory(const char *name, void **p, size_t bytes, int type) {
    if (failing(name)) { *p = NULL; return set(cudaErrorMemoryAllocation); }
    note("alloc", name, (long)bytes);
    for (int i = 0; i < NMEM; i++)
        if (!mem[i].p) {
            *p = mem[i].p = aligned_alloc(4096, (bytes + 8191) / 4096 * 4096);
            memset(*p, 0, bytes);
            mem[i].bytes = bytes, mem[i].type = type;
            return cudaSuccess;
        }
    return set(cudaErrorMemoryAllocation);
}
static cudaError_t give_memory(void *p) {
    for (int i = 0; p && i < NMEM; i++)
        if (mem[i].p == p) { free(p); mem[i].p = NULL; return cudaSuccess; }
    return p ? set(cudaErrorInvalidValue) : cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n) { return get_memory("cudaMalloc", p, n, cudaMemoryTypeDevice); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) { (void)s; return get_memory("cudaMallocAsync", p, n, cudaMemoryTypeDevice); }
cudaError_t cudaMallocManaged(void **p, size_t n, unsigned f) { (void)f; return get_memory("cudaMallocManaged", p, n, cudaMemoryTypeManaged); }
cudaError_t cudaMallocHost(void **p, size_t n) { return get_memory("cudaMallocHost", p, n, cudaMemoryTypeHost); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned f) { (void)f; return get_memory("cudaHostAlloc", p, n, cudaMemoryTypeHost); }
cudaError_t cudaFree(void *p) { return give_memory(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { (void)s; return give_memory(p); }
cudaError_t cudaFreeHost(void *p) { return give_memory(p); }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    for (int i = 0; i < NMEM; i++)
        if (mem[i].p && (const char *)p >= mem[i].p && (const char *)p < mem[i].p + mem[i].bytes) a->type = mem[i].type;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { note("copy", "cudaMemcpy", (long)n); (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t t) { (void)t; note("copy", "cudaMemcpyAsync", (long)n); (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void *d, const void *s, size_t n, size_t o, enum cudaMemcpyKind k) { (void)d; (void)s; (void)n; (void)o; (void)k; return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void *d, const void *s, size_t n, size_t o, enum cudaMemcpyKind k) { (void)s; (void)o; (void)k; memset(d, 0, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s) { (void)s; memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemAdvise(const void *p, size_t n, enum cudaMemoryAdvise a, int d) { (void)p; (void)n; (void)a; (void)d; return cudaSuccess; }
cudaError_t cudaMemPrefetchAsync(const void *p, size_t n, int d, cudaStream_t s) { (void)p; (void)n; (void)d; (void)s; return cudaSuccess; }

static char handles[1 << 16];
static int nhandles;
static void *handle(void) { return handles + ++nhandles; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = handle(); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = handle(); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long f) { (void)g; (void)f; *e = handle(); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = handle(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = handle(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaGetDevice(int *d) { *d = device_now; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device_now = d; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrCooperativeLaunch ? 1 : 0);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return last_error; }
const char *cudaGetErrorString(cudaError_t e) { return e ? "fake error" : "no error"; }

static int encode(void *map, ...) { memset(map, 0, 128); return 0; }
cudaError_t cudaGetDriverEntryPoint(const char *n, void **f, unsigned long long k, enum cudaDriverEntryPointQueryResult *q) {
    (void)n; (void)k;
    *f = (void *)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}

void **__cudaRegisterFatBinary(void *b) { (void)b; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) { (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int t, void *tid, void *bid, void *bd, void *gd, int *w) {
    (void)h; (void)dev; (void)t; (void)tid; (void)bid; (void)bd; (void)gd; (void)w;
    fun[nfun].host = host;
    snprintf(fun[nfun].name, sizeof fun[nfun].name, "%s", name);
    if (nfun < NFUN - 1) nfun++;
}
static int find(const void *f) { int i = 0; while (i < nfun && fun[i].host != f) i++; return i; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fun[find(f)].smem[device_now] = v;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *f) { (void)f; memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t, size_t s, unsigned k) {
    (void)k;
    *n = s > 48 * 1024 && (size_t)fun[find(f)].smem[device_now] < s ? 0 : (t > 256 ? 2 : 3);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t s) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, t, s, 0);
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t s) {
    (void)b; (void)args; (void)s;
    const int i = find(f);
    if (smem > 48 * 1024 && (size_t)fun[i].smem[device_now] < smem) return set(cudaErrorInvalidValue);
    note("launch", fun[i].name, (long)g.x * g.y * g.z);
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t s) {
    return cudaLaunchKernel(f, g, b, args, smem, s);
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *s) {
    call[ncall].grid = g, call[ncall].block = b, call[ncall].smem = smem, call[ncall].s = s;
    ncall++;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
    ncall--;
    *g = call[ncall].grid, *b = call[ncall].block, *smem = call[ncall].smem, *(cudaStream_t *)s = call[ncall].s;
    return cudaSuccess;
}
