// The functions of the CUDA runtime that the library links against (see
// fake_cudart.h).
#include "fake_cudart.h"

#include <sys/syscall.h>
#include <time.h>
#include <unistd.h>

#include <cstdlib>
#include <cstring>

namespace fake {
std::function<cudaError_t()> launch, copy, query, sync;
long long clock_skew_s = 0;
}  // namespace fake

namespace {
cudaError_t g_last = cudaSuccess;
cudaError_t keep(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}
cudaError_t ask(const std::function<cudaError_t()> &f) { return keep(f ? f() : cudaSuccess); }
cudaError_t alloc(void **p, size_t bytes) {
    *p = malloc(bytes);
    memset(*p, 0xA5, bytes);
    return cudaSuccess;
}
char g_dummy[64];
template <typename T>
cudaError_t handle(T *p) {
    *p = (T)(void *)g_dummy;
    return cudaSuccess;
}
}  // namespace

extern "C" {

// std::chrono::steady_clock reads it
int clock_gettime(clockid_t id, struct timespec *t) {
    const int rc = (int)syscall(SYS_clock_gettime, id, t);
    if (id == CLOCK_MONOTONIC) t->tv_sec += fake::clock_skew_s;
    return rc;
}

// what nvcc's host code calls
void **__cudaRegisterFatBinary(void *) { return (void **)g_dummy; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *) { return handle(k); }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) {
    return ask(fake::launch);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
    return ask(fake::launch);
}

// errors
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }

// device
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 0, cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { return *a = *b = 0, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int,
                                                                   size_t, unsigned) {
    return *n = 1, cudaSuccess;
}

// memory
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { return *f = *t = (size_t)1 << 30, cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return alloc(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return alloc(p, n); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
    return alloc(p, n);
}
cudaError_t cudaMallocHost(void **p, size_t n) { return alloc(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return alloc(p, n); }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaFree(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    const cudaError_t e = ask(fake::copy);
    if (e == cudaSuccess) memcpy(d, s, n);
    return e;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    return memset(d, v, n), cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    return memset(a, 0, sizeof *a), cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = g_dummy, cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { return handle(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { return handle(p); }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }

// streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return fake::query ? fake::query() : cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return ask(fake::sync); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
cudaError_t cudaLaunchHostFunc(cudaStream_t, cudaHostFn_t f, void *u) { return f(u), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
    return handle(x);
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"
