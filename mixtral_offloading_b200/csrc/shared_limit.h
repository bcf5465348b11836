// Shared memory beyond 48 KB for kernels whose launches differ in size.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace hqm {

constexpr int SHARED_LIMIT_DEVICES = 64;
// Per kernel: the dynamic shared memory that a launch may ask for on each device (0: not asked yet).
struct SharedLimits {
    std::atomic<int> bytes[SHARED_LIMIT_DEVICES];
};

// True where a launch of `kernel` may use `smem` bytes.  What a kernel is allowed is always all that the device leaves beside
// its static arrays, never the size of the launch at hand: threads whose first launches differ in size then set the same value,
// whichever comes last.
template <typename Kernel>
bool allow_shared(Kernel* kernel, SharedLimits& limits, size_t smem) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int>& have = limits.bytes[dev >= 0 && dev < SHARED_LIMIT_DEVICES ? dev : 0];
    int most = have.load(std::memory_order_acquire);
    if (most == 0) {
        cudaFuncAttributes attr;
        const void* func = reinterpret_cast<const void*>(kernel);
        if (cudaFuncGetAttributes(&attr, func) != cudaSuccess || cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, most -= (int)attr.sharedSizeBytes) != cudaSuccess) {
            cudaGetLastError();
            return false;                                    // (asked again by the next launch)
        }
        have.store(most, std::memory_order_release);
    }
    return smem <= (size_t)most;
}

}  // namespace hqm
