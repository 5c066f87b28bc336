// Dynamic shared memory past 48 KB.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace mcw {

// Lets a kernel take `bytes` of dynamic shared memory on the current device: asked once per device
// and kernel (the attribute is a device's own), and again after a failure.
inline cudaError_t allow_smem(const void *fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> allowed;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    size_t &have = allowed[{dev, fn}];
    if (have >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) have = bytes;
    return e;
}

}  // namespace mcw
