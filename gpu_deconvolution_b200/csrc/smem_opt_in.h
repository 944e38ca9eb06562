// Opt-in of a kernel to large dynamic shared memory.
#pragma once

#include <atomic>
#include <cuda_runtime.h>
#include <stddef.h>

namespace fmvd {

// A launch whose static and dynamic shared memory together pass 48 KB is
// refused until the kernel's limit is raised, per kernel and device.  The limit
// is raised once, to the most that any launch of the kernel asks for: one that
// followed each launch's own size would be lowered by one thread between
// another's opt-in and its launch.  devices: one bit per device that has it.
template <typename K>
cudaError_t allow_smem(K kern, size_t bytes, std::atomic<unsigned long long> &devices)
{
    int dev = 0;
    cudaError_t r = cudaGetDevice(&dev);
    if (r != cudaSuccess)
        return r;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (bit && (devices.load(std::memory_order_acquire) & bit))
        return cudaSuccess;
    r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (r == cudaSuccess)
        devices.fetch_or(bit, std::memory_order_release);
    return r;
}

} // namespace fmvd
