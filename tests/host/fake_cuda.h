// A stand-in for the CUDA runtime calls that a host program of these tests
// goes through (fake_cuda.cpp): device memory is host memory, copies are made at
// once and counted, kernels are recorded and not run.
#pragma once
#include <cuda_runtime.h>
#include <vector>

struct FakeLaunch {
    dim3 grid, block;
};
struct FakeCopy {
    const void* src;
    cudaMemcpyKind kind;
};
extern std::vector<FakeLaunch> fake_launches;
extern std::vector<FakeCopy> fake_copies;   // asynchronous copies and ...
extern size_t fake_waited;                  // ... how many of them a wait has ended
extern int fake_device;                     // the current device
extern bool fake_capture_fails;             // a capture that begins is refused
