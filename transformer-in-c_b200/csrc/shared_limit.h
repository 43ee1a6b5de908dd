// Kernels that need more dynamic shared memory than every launch may ask for.
#pragma once

#include <atomic>
#include <cstdint>
#include <cuda_runtime_api.h>

namespace vitb200 {

// The limit belongs to a kernel on a device.  A process may hold backends on
// several devices one after the other, so a launch site keeps one of these in
// place of a flag and asks it before each launch: the first time on a device it
// raises the limits, afterwards it costs the query of the current device (tens of
// nanoseconds, where setting the attribute takes a few hundred).
class SharedMemoryLimit {
public:
    // False when a limit could not be raised; the next call tries again.
    bool raise(const void *const *kernels, int count, int bytes) {
        int device = -1;
        if (cudaGetDevice(&device) != cudaSuccess || device < 0) {
            return false;
        }
        const uint64_t bit = device < 64 ? uint64_t(1) << device : 0;
        if (raised_.load(std::memory_order_acquire) & bit) {
            return true;
        }
        for (int i = 0; i < count; ++i) {
            if (cudaFuncSetAttribute(kernels[i],
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     bytes) != cudaSuccess) {
                return false;
            }
        }
        raised_.fetch_or(bit, std::memory_order_release);
        return true;
    }
    bool raise(const void *kernel, int bytes) { return raise(&kernel, 1, bytes); }

private:
    std::atomic<uint64_t> raised_{0};   // a bit per device
};

}  // namespace vitb200
