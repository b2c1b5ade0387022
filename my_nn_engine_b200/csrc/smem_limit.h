// The dynamic shared memory that a kernel may ask for is a setting of the kernel on one device.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#include <atomic>

namespace mynn {

// Raises the limit the first time a kernel is launched on a device (a static member of each launcher; a call on every launch took the host
// time that the launch itself takes).  Devices from the 64th on are set each time.
struct SmemLimit {
    std::atomic<uint64_t> done{0};
    cudaError_t raise(const void *kern, size_t bytes) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = dev < 64 ? 1ull << dev : 0;
        if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

}  // namespace mynn
