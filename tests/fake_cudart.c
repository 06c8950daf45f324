/* A CUDA runtime without a GPU for tests of the library's host code: device
 * memory is host memory, kernels are counted and do nothing, and the test says
 * what fails, which stream is being captured and when the context is reset.
 * Linked in place of libcudart (tests/test_host_runtime.py). */
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

static size_t g_limit = (size_t)1 << 30;
static int g_launches, g_fail_launch = -1, g_host_allocs, g_symbols, g_attributes;
static cudaStream_t g_capturing;
static int g_any_capture;
static unsigned long long g_context = 1;
static struct { dim3 grid, block; size_t smem; void *stream; } g_call;

/* --- what a test controls and reads ------------------------------------- */
void fake_limit(size_t bytes) { g_limit = bytes; }             /* larger device allocations fail */
void fake_fail_launch(int after) { g_fail_launch = after; }    /* the launch after that many fails; -1: none */
void fake_capture(int on, void *stream) { g_any_capture = on; g_capturing = (cudaStream_t)stream; }
void fake_new_context(void) { g_context++; }                   /* as after cudaDeviceReset */
int fake_launches(void) { return g_launches; }
int fake_host_allocs(void) { return g_host_allocs; }
int fake_symbol_lookups(void) { return g_symbols; }
int fake_attributes(void) { return g_attributes; }

/* --- registration ---------------------------------------------------------- */
void **__cudaRegisterFatBinary(void *f) { (void)f; static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *f, char *d, const char *n, int t, uint3 *a, uint3 *b, dim3 *c, dim3 *e,
                            int *w) {
    (void)h; (void)f; (void)d; (void)n; (void)t; (void)a; (void)b; (void)c; (void)e; (void)w;
}
void __cudaRegisterVar(void **h, char *v, char *d, const char *n, int e, size_t s, int c, int g) {
    (void)h; (void)v; (void)d; (void)n; (void)e; (void)s; (void)c; (void)g;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream) {
    g_call.grid = grid; g_call.block = block; g_call.smem = smem; g_call.stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = g_call.grid; *block = g_call.block; *smem = g_call.smem; *(void **)stream = g_call.stream;
    return cudaSuccess;
}

/* --- memory ----------------------------------------------------------------- */
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = NULL;
    if (n > g_limit) return cudaErrorMemoryAllocation;
    return posix_memalign(p, 256, n ? n : 1) ? cudaErrorMemoryAllocation : (memset(*p, 0, n), cudaSuccess);
}
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned flags) {
    (void)flags;
    g_host_allocs++;
    *p = calloc(1, n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) {
    (void)k;
    if (n && (!d || (size_t)s < 4096)) return cudaErrorInvalidValue;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
    if (n && (size_t)d < 4096) return cudaErrorInvalidValue;
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { (void)st; return cudaMemset(d, v, n); }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { g_symbols++; *p = (void *)s; return cudaSuccess; }

/* --- launches ----------------------------------------------------------------- */
static cudaError_t launch(void) { return g_launches++ == g_fail_launch ? cudaErrorLaunchOutOfResources : cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t s, cudaStream_t st) {
    (void)f; (void)g; (void)b; (void)a; (void)s; (void)st;
    return launch();
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a) {
    (void)c; (void)f; (void)a;
    return launch();
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
    (void)f; (void)a; (void)v;
    g_attributes++;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
    (void)f; (void)b; (void)s; (void)fl;
    *n = 2;
    return cudaSuccess;
}

/* --- device, streams, events, graphs ------------------------------------------- */
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(struct cudaDeviceProp *p, int d) {
    (void)d;
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
static CUresult ctx_get_id(CUcontext c, unsigned long long *id) { (void)c; *id = g_context; return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char *name, void **fn, unsigned long long flags,
                                    enum cudaDriverEntryPointQueryResult *q) {
    (void)flags;
    *fn = strcmp(name, "cuCtxGetId") == 0 ? (void *)ctx_get_id : NULL; /* no tensor maps */
    if (q) *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return *fn ? cudaSuccess : cudaErrorSymbolNotFound;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *st) {
    *st = g_any_capture && s == g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)malloc(1); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long f) {
    (void)g; (void)f;
    *e = (cudaGraphExec_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 1.f; return cudaSuccess; }
