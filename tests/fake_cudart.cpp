// A CUDA runtime for the launching code alone: it answers what a test asks for
// and launches nothing.
#include <cuda_runtime_api.h>

extern "C" {
int fake_device, fake_attribute_answer, fake_launch_answer, fake_launches;

cudaError_t cudaGetDevice(int *d) {
    *d = fake_device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return (cudaError_t)fake_attribute_answer; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
    ++fake_launches;
    return (cudaError_t)fake_launch_answer;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
    ++fake_launches;
    return (cudaError_t)fake_launch_answer;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }

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
cudaError_t __cudaGetKernel(void **, const void *) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(void *, dim3, dim3, void **, size_t, cudaStream_t) {
    ++fake_launches;
    return (cudaError_t)fake_launch_answer;
}
}
