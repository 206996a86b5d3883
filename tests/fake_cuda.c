/* A CUDA runtime without a device: the calls libhsflow's host code makes, each recorded as one line
 * of text.  Kernels do not run.  tests/fake_cuda.py links the library's objects against this file. */
#include <cuda_runtime_api.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static struct { const void *host; const char *name; } kernels[4096];
static int nkernels;
static char *text;
static size_t len, cap;
static int coop_limit = 1 << 30; /* cooperative launches of more blocks are refused */
static int held = 16; /* warps of any kernel that an SM holds at once */
static int queries; /* calls that ask for the device or an attribute */

static void record(const char *fmt, ...) {
    va_list ap;
    if (cap - len < 512) text = realloc(text, cap = 2 * cap + 4096);
    va_start(ap, fmt);
    len += vsnprintf(text + len, cap - len, fmt, ap);
    va_end(ap);
}
static const char *name_of(const void *host) {
    for (int i = 0; i < nkernels; ++i)
        if (kernels[i].host == host) return kernels[i].name;
    return "?";
}

void fake_reset(int max_cooperative_blocks) {
    len = 0;
    queries = 0;
    coop_limit = max_cooperative_blocks;
    record("%s", "");
}
void fake_hold(int warps) { held = warps; }
const char *fake_log(void) { return text ? text : ""; }
int fake_queries(void) { return queries; }

/* registration and launches */
void **__cudaRegisterFatBinary(void *p) { static void *h; (void)p; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) { (void)h; }
void __cudaUnregisterFatBinary(void **h) { (void)h; }
void __cudaRegisterVar(void **h, char *v, char *a, const char *n, int e, size_t s, int c, int g) {
    (void)h; (void)v; (void)a; (void)n; (void)e; (void)s; (void)c; (void)g;
}
void __cudaRegisterFunction(void **h, const char *host, char *dev, const char *name, int limit, void *tid, void *bid,
                            void *bdim, void *gdim, int *ws) {
    (void)h; (void)dev; (void)limit; (void)tid; (void)bid; (void)bdim; (void)gdim; (void)ws;
    if (nkernels < 4096) { kernels[nkernels].host = host; kernels[nkernels++].name = name; }
}
static struct { dim3 grid, block; size_t smem; void *stream; } pushed;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *s) {
    pushed.grid = grid; pushed.block = block; pushed.smem = smem; pushed.stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
    *grid = pushed.grid; *block = pushed.block; *smem = pushed.smem; *(void **)s = pushed.stream;
    return cudaSuccess;
}
/* launch: mangled name, grid, threads of a block, the first 8 bytes of the first argument */
static cudaError_t launch(const char *what, const void *f, dim3 g, dim3 b, void **args) {
    uint64_t first = 0;
    memcpy(&first, args[0], sizeof first);
    record("%s %s %u %u %u %u %llu\n", what, name_of(f), g.x, g.y, g.z, b.x * b.y * b.z, (unsigned long long)first);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t s) {
    (void)smem; (void)s;
    return launch("launch", f, g, b, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) {
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeCooperative && c->attrs[i].val.cooperative &&
            (int)c->gridDim.x > coop_limit) {
            launch("refused", f, c->gridDim, c->blockDim, args);
            return cudaErrorCooperativeLaunchTooLarge;
        }
    return launch("launch", f, c->gridDim, c->blockDim, args);
}

/* memory and queries */
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
    (void)s;
    record("memset %llu %d %zu\n", (unsigned long long)(uintptr_t)p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *p, size_t n, enum cudaMemcpyKind k, cudaStream_t s) {
    (void)k; (void)s;
    record("memcpy %llu %llu %zu\n", (unsigned long long)(uintptr_t)d, (unsigned long long)(uintptr_t)p, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *p, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k,
                              cudaStream_t s) {
    (void)dp; (void)sp;
    return cudaMemcpyAsync(d, p, w * h, k, s);
}
cudaError_t cudaGetDevice(int *d) { ++queries; *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10 : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
    (void)f; (void)a; (void)v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
    (void)f; (void)s; (void)fl;
    ++queries;
    *n = held / (b / 32);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int b, size_t s) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, b, s, 0);
}
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) { (void)sym; *p = (void *)(uintptr_t)0x7000000000; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; *s = (cudaStream_t)(uintptr_t)1; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) {
    (void)s;
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; *e = (cudaEvent_t)(uintptr_t)1; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { (void)e; (void)s; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { (void)e; return "fake"; }
cudaError_t cudaLibraryLoadData(cudaLibrary_t *l, const void *c, enum cudaJitOption *jo, void **jv, unsigned nj,
                                enum cudaLibraryOption *lo, void **lv, unsigned nl) {
    (void)l; (void)c; (void)jo; (void)jv; (void)nj; (void)lo; (void)lv; (void)nl;
    return cudaErrorNotSupported;
}
cudaError_t cudaLibraryGetKernel(cudaKernel_t *k, cudaLibrary_t l, const char *n) {
    (void)k; (void)l; (void)n;
    return cudaErrorNotSupported;
}
