// The limit of a kernel's dynamic shared memory. It belongs to the current device's copy of the kernel: raised on one device, a launch
// that needs it still fails on another. Host code alone, no device code.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>

namespace stride {

// Raises KERNEL's limit to `bytes`, once a device. `bytes` is the most that any call asks for: a limit that followed the calls could be
// lowered by one thread between another's call and its launch.
template <auto KERNEL>
inline cudaError_t allow_shared(int bytes) {
    static std::atomic<bool> done[64] = {};
    int device = 0;
    const cudaError_t found = cudaGetDevice(&device);
    if (found != cudaSuccess) return found;
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    if (done[device].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(KERNEL), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done[device].store(true, std::memory_order_release);
    return e;
}

}  // namespace stride
