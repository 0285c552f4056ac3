// A stand-in for the CUDA runtime calls that a host program of these tests
// goes through: kernels are recorded and not run.
#pragma once
#include <cuda_runtime.h>
#include <vector>

struct FakeLaunch {
    dim3 grid, block;
};
static std::vector<FakeLaunch> fake_launches;

extern "C" {
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void*) {
    *kernel = nullptr;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3 grid, dim3 block, void**, size_t, cudaStream_t) {
    fake_launches.push_back({grid, block});
    return cudaSuccess;
}
}
