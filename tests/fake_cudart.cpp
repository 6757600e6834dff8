// A CUDA runtime without a GPU, for the code that calls it: device memory is
// host memory full of ones, which kernels (never run) and memset leave alone,
// copies copy, and a test says which calls are refused.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <unordered_map>

extern "C" {
int fake_device, fake_attribute_answer;
int fake_launch_answer;   // of cudaLaunchKernelEx (sweeps and cooperative runs)
int fake_launches;        // how many of those were asked for
int fake_sync_failures;   // so many waits fail after the first of those launches
void (*fake_on_occupancy)(int call);  // called by the occupancy query of clusters, with its number
int fake_occupancy_calls;
size_t fake_used, fake_peak;  // bytes of device memory
size_t fake_limit;            // the most that can be had (0: any)

static void *ones(size_t bytes) {
    double *p = (double *)malloc(bytes + 256);
    for (size_t i = 0; i < (bytes + 7) / 8; ++i) p[i] = 1.0;
    return p;
}

cudaError_t cudaGetDevice(int *d) {
    *d = fake_device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    fake_device = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return (cudaError_t)fake_attribute_answer; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
    *n = 16;
    const int call = ++fake_occupancy_calls;
    if (fake_on_occupancy) fake_on_occupancy(call);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
    ++fake_launches;
    return (cudaError_t)fake_launch_answer;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "refused by the test"; }

static std::unordered_map<void *, size_t> &sizes() {
    static auto *m = new std::unordered_map<void *, size_t>;
    return *m;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    if (fake_limit && fake_used + n > fake_limit) return cudaErrorMemoryAllocation;
    *p = ones(n);
    sizes()[*p] = n;
    fake_used += n;
    if (fake_used > fake_peak) fake_peak = fake_used;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (p) {
        fake_used -= sizes()[p];
        sizes().erase(p);
    }
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = ones(n);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void *p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *, const cudaMemPoolProps *) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
    *f = *t = (size_t)1 << 36;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t i = 0; i < h; ++i) memmove((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorNotSupported; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }

cudaError_t cudaStreamCreate(cudaStream_t *s) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return cudaStreamCreate(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    if (fake_launches > 0 && fake_sync_failures > 0) {
        --fake_sync_failures;
        return cudaErrorUnknown;
    }
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long, cudaDriverEntryPointQueryResult *) {
    return cudaErrorNotSupported;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}

// What objects of compiled kernels register and call.
void **__cudaRegisterFatBinary(void *) {
    static void *h[1];
    return h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
char __cudaInitModule(void **) { return 1; }
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
}
