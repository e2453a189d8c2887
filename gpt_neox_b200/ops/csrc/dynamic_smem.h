// Dynamic shared memory above 48 KB has to be allowed for a kernel, and the permission belongs to the device that is current
// when it is given: a process that uses two devices gives it on both.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

// Allows `bytes` (always the same for one kernel) on the current device; asks the runtime once per kernel and device.
template <auto KERNEL>
inline bool allow_dynamic_smem(size_t bytes) {
    static std::atomic<unsigned long long> allowed{0};          // one bit per device; devices past the 64th ask every time
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (allowed.load(std::memory_order_relaxed) & bit) return true;
    if (cudaFuncSetAttribute(reinterpret_cast<const void*>(KERNEL), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) !=
        cudaSuccess)
        return false;
    allowed.fetch_or(bit, std::memory_order_relaxed);
    return true;
}
