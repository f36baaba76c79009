// Dynamic shared memory beyond 48 KB.
//
// The limit of a launch is an attribute of the function, shared by every context and host thread of the process.  Set
// to what the launch at hand needs, it could be lowered by another thread between this thread's setting and its launch,
// which is then refused; so it is only ever set to one value, the most that the device gives the kernel.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

namespace qpd {

// Let K be launched with `bytes` of dynamic shared memory on the current device.
template <auto K> cudaError_t allow_smem(size_t bytes) {
    static std::atomic<int> fixed{-1};  // bytes of the kernel's own static shared memory
    int own = fixed.load(std::memory_order_relaxed);
    if (own < 0) {
        cudaFuncAttributes at;
        const cudaError_t e = cudaFuncGetAttributes(&at, K);
        if (e != cudaSuccess) return e;
        own = (int)at.sharedSizeBytes;
        fixed.store(own, std::memory_order_relaxed);
    }
    if (bytes + own <= 48 * 1024) return cudaSuccess;
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    if (bytes + own > (size_t)optin) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - own);
}

}  // namespace qpd
