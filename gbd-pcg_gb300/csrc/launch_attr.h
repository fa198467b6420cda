// Limits of a kernel's launches.  They belong to the function on its device, so
// every handle and thread of the process shares them.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace gbdpcg {

// Lets `func` be launched with `bytes` of dynamic shared memory on the current
// device.  The limit is only raised: a call that set its own need could lower it
// between another thread's call and that thread's launch, which would be refused.
inline cudaError_t allow_dynamic_smem(const void *func, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> limits;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    size_t &limit = limits[{device, func}];
    if (bytes <= limit) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) limit = bytes;
    return e;
}

}  // namespace gbdpcg
