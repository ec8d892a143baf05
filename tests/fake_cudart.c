/* fake_cudart.c — the CUDA runtime calls the library makes, over host memory: device buffers are heap blocks, copies are
 * memcpy, a kernel launch runs nothing. Linked with the library's own archive (fake_cuda.py) it lets a test follow the host
 * side without a GPU: every launch, copy and synchronisation is told to a hook, which may answer with an error code. */
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

/* what: "launch", "memcpy", "sync"; name: the kernel's; a: its arguments / the destination; b: the source; n: grid.x / bytes */
typedef int (*fake_hook)(const char *what, const char *name, void *a, const void *b, size_t n, void *stream);
static fake_hook hook;
static int sms = 148;
void fake_set_hook(fake_hook h) { hook = h; }
void fake_set_sms(int n) { sms = n; }

static struct { const void *fn; const char *name; } kernels[1024];
static int n_kernels;
static const char *name_of(const void *fn) {
    for (int i = 0; i < n_kernels; i++) if (kernels[i].fn == fn) return kernels[i].name;
    return "?";
}
static cudaError_t tell(const char *what, const char *name, void *a, const void *b, size_t n, void *stream) {
    return hook ? (cudaError_t)hook(what, name, a, b, n, stream) : cudaSuccess;
}
static _Thread_local cudaError_t last;
static cudaError_t keep(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }

/* ---- what the compiler's host code calls */
static void *module_handle[1];
void **__cudaRegisterFatBinary(void *bin) { (void)bin; return module_handle; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int limit, uint3 *t, uint3 *b, dim3 *bd, dim3 *gd, int *w) {
    (void)h; (void)dev; (void)limit; (void)t; (void)b; (void)bd; (void)gd; (void)w;
    if (n_kernels < 1024) { kernels[n_kernels].fn = host; kernels[n_kernels++].name = name; }
}
void __cudaRegisterVar(void **h, char *host, char *dev, const char *name, int ext, size_t size, int constant, int global) {
    (void)h; (void)host; (void)dev; (void)name; (void)ext; (void)size; (void)constant; (void)global;
}
static _Thread_local struct { dim3 g, b; size_t smem; void *st; } pushed;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *st) { pushed.g = g; pushed.b = b; pushed.smem = smem; pushed.st = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) { *g = pushed.g; *b = pushed.b; *smem = pushed.smem; *(void **)st = pushed.st; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t st) { (void)b; (void)smem; return keep(tell("launch", name_of(f), args, NULL, g.x, st)); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) { return keep(tell("launch", name_of(f), args, NULL, c->gridDim.x, c->stream)); }

/* ---- memory */
static cudaError_t take(void **p, size_t n) { *p = aligned_alloc(256, (n + 255) & ~(size_t)255); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)k;
    const cudaError_t e = tell("memcpy", "", d, s, n, st);
    if (e == cudaSuccess) memcpy(d, s, n);
    return keep(e);
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k, cudaStream_t st) {
    (void)k; (void)st;
    for (size_t i = 0; i < h; i++) memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t st) { (void)st; memset(p, v, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) { (void)sym; return take(p, 1 << 16); }

/* ---- device, streams, events, graphs */
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d == 0 ? cudaSuccess : cudaErrorInvalidDevice; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? sms : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int d) { (void)d; memset(p, 0, sizeof *p); p->major = 10; p->multiProcessorCount = sms; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return tell("sync", "", NULL, NULL, 0, NULL); }
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { (void)e; return "error of the fake runtime"; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { (void)f; (void)a; (void)v; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *f) { (void)f; memset(a, 0, sizeof *a); a->numRegs = 72; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)malloc(16); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free((void *)s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return tell("sync", "", NULL, NULL, 0, s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)module_handle; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *v) { (void)s; *v = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f) { (void)g; (void)f; *x = (cudaGraphExec_t)module_handle; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { (void)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { (void)x; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)module_handle; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t *h, void *p) { (void)h; (void)p; return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void **p, cudaIpcMemHandle_t h, unsigned f) { (void)p; (void)h; (void)f; return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void *p) { (void)p; return cudaErrorNotSupported; }

static CUresult encode_tiled(CUtensorMap *m, CUtensorMapDataType t, cuuint32_t rank, void *p, const cuuint64_t *dim, const cuuint64_t *stride, const cuuint32_t *box,
                             const cuuint32_t *es, CUtensorMapInterleave il, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2, CUtensorMapFloatOOBfill oob) {
    (void)t; (void)dim; (void)box; (void)es; (void)il; (void)sw; (void)l2; (void)oob;
    if ((size_t)p & 15) return CUDA_ERROR_INVALID_VALUE;
    for (cuuint32_t i = 0; i + 1 < rank; i++) if (stride[i] & 15) return CUDA_ERROR_INVALID_VALUE;
    memset(m, 0, sizeof *m);
    return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPoint(const char *sym, void **fn, unsigned long long flags, enum cudaDriverEntryPointQueryResult *q) {
    (void)flags;
    *fn = strcmp(sym, "cuTensorMapEncodeTiled") ? NULL : (void *)encode_tiled;
    if (q) *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
