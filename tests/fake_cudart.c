/* A CUDA runtime without a GPU, for tests of the library's host side: memory is
 * host memory, kernels do nothing, graphs are counters, and chosen calls fail
 * with an error code (and leave it as the last error, as the runtime does).
 * Only what the library calls is here. */
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#define API __attribute__((visibility("default")))

enum { CALL_LAUNCH, CALL_ATTRIBUTE, CALL_CLUSTERS, CALL_HOST_ALLOC, CALL_SYNC, CALL_KINDS };

static cudaError_t last_error = cudaSuccess;
static long calls[CALL_KINDS];
static long fail_at[CALL_KINDS] = {-1, -1, -1, -1, -1}; /* index of the call that fails, -1: none */
static long open_captures, live_graphs, graph_launches, unprobed_clusters;
static const void* probed[16]; /* kernels that occupancy was asked for, in clusters */
static int probes;
static struct { const void* kernel; unsigned grid, block; } launched[256]; /* since the reset */
static int sms = 148;

static cudaError_t done(cudaError_t e) {
    if (e != cudaSuccess) last_error = e;
    return e;
}
static cudaError_t counted(int kind, cudaError_t e) {
    return done(calls[kind]++ == fail_at[kind] ? e : cudaSuccess);
}

/* for the tests */
API void fake_reset(void) {
    for (int k = 0; k < CALL_KINDS; ++k) calls[k] = 0, fail_at[k] = -1;
    last_error = cudaSuccess;
    unprobed_clusters = 0;
}
API void fake_forget_probes(void) { probes = 0; }
API void fake_set_sms(int n) { sms = n; }
API const void* fake_launched(int k) { return launched[k].kernel; }
API unsigned fake_grid(int k) { return launched[k].grid; }
API unsigned fake_block(int k) { return launched[k].block; }
API void fake_fail(int kind, long index) { fail_at[kind] = index; }
API long fake_calls(int kind) { return calls[kind]; }
API int fake_last_error(void) { return last_error; }
API long fake_open_captures(void) { return open_captures; }
API long fake_live_graphs(void) { return live_graphs; }
API long fake_graph_launches(void) { return graph_launches; }
/* launches of a cluster of blocks whose kernel has not been asked for */
API long fake_unprobed_clusters(void) { return unprobed_clusters; }

/* what compiled .cu objects register */
void** __cudaRegisterFatBinary(void* f) { (void)f; return calloc(1, sizeof(void*)); }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { free(h); }
void __cudaRegisterFunction(void** h, const char* f, char* d, const char* n, int l, uint3* t, uint3* b,
                            dim3* bd, dim3* gd, int* w) {
    (void)h, (void)f, (void)d, (void)n, (void)l, (void)t, (void)b, (void)bd, (void)gd, (void)w;
}
void __cudaRegisterVar(void** h, char* v, char* d, const char* n, int e, size_t s, int c, int g) {
    (void)h, (void)v, (void)d, (void)n, (void)e, (void)s, (void)c, (void)g;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
    (void)g, (void)b, (void)s, (void)st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    *g = (dim3){1, 1, 1}, *b = (dim3){1, 1, 1}, *s = 0, *(void**)st = NULL;
    return cudaSuccess;
}

/* launches */
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t s, cudaStream_t st) {
    (void)f, (void)g, (void)b, (void)a, (void)s, (void)st;
    return counted(CALL_LAUNCH, cudaErrorLaunchOutOfResources);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
    (void)a;
    if (calls[CALL_LAUNCH] < 256) {
        launched[calls[CALL_LAUNCH]].kernel = f;
        launched[calls[CALL_LAUNCH]].grid = c->gridDim.x;
        launched[calls[CALL_LAUNCH]].block = c->blockDim.x;
    }
    for (unsigned k = 0; k < c->numAttrs; ++k)
        if (c->attrs[k].id == cudaLaunchAttributeClusterDimension) {
            int known = 0;
            for (int q = 0; q < probes; ++q) known |= probed[q] == f;
            unprobed_clusters += !known;
        }
    return counted(CALL_LAUNCH, cudaErrorLaunchOutOfResources);
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
    (void)f, (void)a, (void)v;
    return counted(CALL_ATTRIBUTE, cudaErrorInvalidValue);
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    (void)c;
    if (probes < 16) probed[probes++] = f;
    *n = 0;
    const cudaError_t e = counted(CALL_CLUSTERS, cudaErrorInvalidClusterSize);
    if (e == cudaSuccess) *n = 8;
    return e;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int b,
                                                                   size_t s, unsigned fl) {
    (void)f, (void)b, (void)s, (void)fl;
    *n = 4;
    return cudaSuccess;
}

/* errors and devices */
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e ? "the fake's error" : "no error"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
    (void)a, (void)d;
    *v = sms;
    return cudaSuccess;
}

/* memory */
cudaError_t cudaMalloc(void** p, size_t n) {
    return done((*p = calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) {
    (void)f;
    const cudaError_t e = counted(CALL_HOST_ALLOC, cudaErrorMemoryAllocation);
    return e == cudaSuccess ? cudaMalloc(p, n) : e;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
    (void)k;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h,
                         enum cudaMemcpyKind k) {
    (void)k;
    for (size_t r = 0; r < h; ++r) memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    (void)st;
    return cudaMemset(d, v, n);
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
    static void* symbol;  /* the library has one device variable, below 8 MB */
    (void)s;
    if (!symbol) symbol = calloc(1, 8 << 20);
    *p = symbol;
    return cudaSuccess;
}

/* streams, events, graphs */
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
    (void)f;
    *s = (cudaStream_t)calloc(1, 8);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    (void)s;
    return counted(CALL_SYNC, cudaErrorLaunchFailure);
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
    (void)s, (void)e, (void)f;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) {
    (void)s, (void)m;
    if (open_captures) return done(cudaErrorIllegalState);
    ++open_captures;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    (void)s;
    --open_captures;
    ++live_graphs;
    *g = (cudaGraph_t)calloc(1, 8);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { --live_graphs; free(g); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long f) {
    (void)g, (void)f;
    *x = (cudaGraphExec_t)calloc(1, 8);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
    (void)x, (void)s;
    ++graph_launches;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e, (void)s; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
    (void)a, (void)b;
    *ms = 1.f;
    return cudaSuccess;
}
