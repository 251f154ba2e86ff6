// The shared memory that a kernel may ask for is an attribute of it on one device: it is set once per device, and not until it succeeds does
// a device count as done.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>

namespace mb {

using DeviceSet = std::atomic<unsigned long long>;  // a bit per device; devices beyond the 64th are set at every launch

inline cudaError_t reserve_on_device(const void* kernel, int bytes, DeviceSet& done) {
    int device = 0;
    cudaError_t status = cudaGetDevice(&device);
    if (status != cudaSuccess) return status;
    const unsigned long long bit = device < 64 ? 1ull << device : 0;
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (status == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
    return status;
}

}  // namespace mb
