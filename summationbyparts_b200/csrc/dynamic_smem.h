// Opt-in of a kernel to more than the default 48 KB of dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace sbp {

// One per kernel.  The attribute belongs to the function on one device, so what has been set is kept per
// device (of the first 64; on others it is set for every launch).  Safe from several threads: at worst
// two set the same value.
class DynamicSmem {
    std::atomic<uint64_t> devices_{0};

public:
    // Allows `bytes` (the same for every call) on the current device.
    cudaError_t allow(const void* kernel, size_t bytes) {
        int d = 0;
        const cudaError_t e = cudaGetDevice(&d);
        if (e != cudaSuccess) return e;
        const uint64_t bit = d < 64 ? uint64_t(1) << d : 0;
        if (devices_.load(std::memory_order_relaxed) & bit) return cudaSuccess;
        const cudaError_t s = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (s == cudaSuccess) devices_.fetch_or(bit, std::memory_order_relaxed);
        return s;
    }
};

}  // namespace sbp
