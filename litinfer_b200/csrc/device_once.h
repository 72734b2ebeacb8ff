// What a launcher has to ask or tell the driver once on every device: a kernel's limit of dynamic shared memory belongs to the
// device that was current when it was raised, and so does a count of multiprocessors.  Marks are per device, so that a process
// that uses several finds each of them set up; two threads that meet on a first call do it twice, which changes nothing.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstddef>

constexpr int kLiDevices = 64;          // devices with a mark of their own; on any further one it is done on every call

struct LiOncePerDevice {
    std::atomic<unsigned char> done[kLiDevices] = {};
};

// Raises the dynamic shared memory of `kernel` to `bytes` on the current device.
static inline cudaError_t li_raise_shared(LiOncePerDevice& once, const void* kernel, size_t bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool marked = dev >= 0 && dev < kLiDevices;
    if (marked && once.done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && marked) once.done[dev].store(1, std::memory_order_release);
    return e;
}

// Multiprocessors of the current device (148 if it cannot be asked).
inline int li_multiprocessors() {
    static std::atomic<int> count[kLiDevices] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 148;
    if (dev < kLiDevices && (n = count[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    if (dev < kLiDevices) count[dev].store(n, std::memory_order_relaxed);
    return n;
}
