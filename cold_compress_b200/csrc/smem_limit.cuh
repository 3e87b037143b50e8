// smem_limit.cuh -- how much dynamic shared memory a kernel may be launched with.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

// Beside its static arrays a kernel has up to 48 KB unless more is allowed, for each kernel and on each device.  One of these per kernel,
// static.  It allows what the device has, once: threads that launch the kernel with different sizes then do not take back
// from one another what they need.  A failure is not remembered.
class SmemLimit {
    std::atomic<uint64_t> devices{0};

  public:
    cudaError_t allow(const void* kernel, size_t smem) {
        if (smem <= 4 * 1024) return cudaSuccess;      // static arrays: 42 KB at most
        int dev = 0, most = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = dev < 64 ? 1ull << dev : 0;
        if (devices.load(std::memory_order_relaxed) & bit) return cudaSuccess;
        cudaFuncAttributes own;
        if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
        if ((e = cudaFuncGetAttributes(&own, kernel)) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)own.sharedSizeBytes)) != cudaSuccess) return e;
        devices.fetch_or(bit, std::memory_order_relaxed);
        return cudaSuccess;
    }
    template <typename... A>
    cudaError_t allow(void (*kernel)(A...), size_t smem) { return allow((const void*)kernel, smem); }
};
