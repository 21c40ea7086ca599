// gb_once.h — host settings that belong to a device.
#pragma once
#include <atomic>
#include <cuda_runtime_api.h>
#include <stdint.h>

namespace gb {

// What a process sets once for each device (a kernel's shared-memory limit is
// one device's): f runs until it has succeeded on the current one.
struct OncePerDevice {
    std::atomic<uint64_t> done{0};
    template <class F>
    cudaError_t operator()(F f) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e) return e;
        const uint64_t bit = dev < 64 ? 1ull << dev : 0;  // past 64 devices: each time
        if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
        if ((e = f()) == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

}  // namespace gb
