// Opt-in of a kernel to more than 48 KB of dynamic shared memory: an attribute of the kernel on each device, set once.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace ftb200 {

constexpr int kDevicesKnown = 64;  // devices above are served too, with the attribute set on every call

// `done` belongs to the kernel.  Two threads may both set the attribute: the value is the same.
template<class F>
inline cudaError_t opt_in_smem(F kernel, size_t bytes, std::atomic<bool> (&done)[kDevicesKnown])
{
    int               dev = 0;
    const cudaError_t e   = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    const bool known = dev >= 0 && dev < kDevicesKnown;
    if (known && done[dev].load(std::memory_order_acquire)) {
        return cudaSuccess;
    }
    const cudaError_t f = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (f == cudaSuccess && known) {
        done[dev].store(true, std::memory_order_release);
    }
    return f;
}

// The same for a kernel whose need moves with the call: the attribute is only ever raised, because another thread may stand
// between its look at the occupancy and its launch.  `highest` belongs to the kernel and the current device; under a lock.
template<class F>
inline cudaError_t raise_smem(F kernel, size_t bytes, size_t& highest)
{
    if (bytes <= highest) {
        return cudaSuccess;
    }
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) {
        highest = bytes;
    }
    return e;
}

}  // namespace ftb200
