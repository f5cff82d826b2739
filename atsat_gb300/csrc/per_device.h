// What belongs to a device and is kept for the process: handles may live on several devices, in several threads. Every
// call here is about the current device (each entry point makes its handle's device current).
#pragma once

#include <atomic>
#include <cstddef>

#include <cuda_runtime_api.h>

namespace atsat {

constexpr int KEPT_DEVICES = 64;       // devices beyond are asked each time

// the current device, -1 where there is none
inline int current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return dev;
}

// SMs of the current device
inline int sm_count() {
    static std::atomic<int> known[KEPT_DEVICES];
    const int dev = current_device();
    const bool kept = dev >= 0 && dev < KEPT_DEVICES;
    int n = kept ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n > 0) return n;
    if (dev < 0 || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
        cudaGetLastError();
        return 152;
    }
    if (kept) known[dev].store(n, std::memory_order_relaxed);
    return n;
}

// Lets a kernel have more dynamic shared memory than a launch gets by default. The limit is the kernel's on one device,
// so it is set once for each (a function-local static of the launch that needs it).
class SharedMemory {
public:
    cudaError_t allow(const void* kernel, size_t bytes) {
        const int dev = current_device();
        const bool kept = dev >= 0 && dev < KEPT_DEVICES;
        if (kept && done_[dev].load(std::memory_order_relaxed)) return cudaSuccess;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess && kept) done_[dev].store(true, std::memory_order_relaxed);
        return e;
    }

private:
    std::atomic<bool> done_[KEPT_DEVICES] = {};
};

}  // namespace atsat
