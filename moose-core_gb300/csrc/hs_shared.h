// hs_shared.h -- dynamic shared memory of the stepping kernels.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <utility>
#include <vector>

namespace hsg {

// Lets `kernel` (a __global__ function) take as much dynamic shared memory as
// the current device has for it beside its static arrays.  The attribute is
// the function's, not the launch's, and shared by every thread of the process:
// set to what one launch needs, it would refuse another thread's larger one in
// between.  So it is set once per kernel and device, and a launch's own size
// decides what it takes.
inline cudaError_t allowShared(const void* kernel) {
    static std::mutex lock;
    static std::vector<std::pair<const void*, int>> done;
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> hold(lock);
    for (const auto& d : done)
        if (d.first == kernel && d.second == dev) return cudaSuccess;
    cudaFuncAttributes a;
    e = cudaFuncGetAttributes(&a, kernel);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes);
    if (e == cudaSuccess) done.push_back({kernel, dev});
    return e;
}

}  // namespace hsg
