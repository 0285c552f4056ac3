#include "fake_cuda.h"
#include <stdlib.h>
#include <string.h>

std::vector<FakeLaunch> fake_launches;
std::vector<FakeCopy> fake_copies;
size_t fake_waited = 0;
int fake_device = 0;
bool fake_capture_fails = false;

extern "C" {
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void*) {
    *kernel = nullptr;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3 grid, dim3 block, void**, size_t, cudaStream_t) {
    fake_launches.push_back({grid, block});
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* dev) {
    *dev = fake_device;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) {
    *value = 0;   // the callers' fallbacks
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { return (*p = calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind) {
    memcpy(dst, src, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    memcpy(dst, src, n);
    fake_copies.push_back({src, kind});
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    memset(p, v, n);
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    fake_waited = fake_copies.size();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    return fake_capture_fails ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = nullptr;
    return cudaSuccess;
}
