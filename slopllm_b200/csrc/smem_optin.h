// Shared memory beyond 48 KB: a kernel's attributes belong to one device, and are set there at its first launch.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>

// One static object per kernel, at the place that launches it.  Any thread, any device; what failed is tried again at the next launch.
class SmemOptIn {
public:
    // 0, or the error with which the launch must not go on.  `carveout` (per cent of the SM's memory): negative, as the driver chooses.
    int operator()(const void* kernel, int bytes, int carveout = -1) {
        int device = 0;
        cudaError_t rc = cudaGetDevice(&device);
        const uint64_t bit = rc == cudaSuccess && device < 64 ? 1ull << device : 0;
        if ((done_.load(std::memory_order_acquire) & bit) != 0) return 0;
        if (rc == cudaSuccess) rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (rc == cudaSuccess && carveout >= 0) rc = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
        if (rc != cudaSuccess) {
            cudaGetLastError();
            return (int)rc;
        }
        done_.fetch_or(bit, std::memory_order_release);
        return 0;
    }

private:
    std::atomic<uint64_t> done_{0};
};
