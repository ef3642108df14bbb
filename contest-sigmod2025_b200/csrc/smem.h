// Leave for a kernel to take more dynamic shared memory than the 48 KiB that
// every launch may have.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstddef>
#include <cstdint>

namespace bj {

// Before a launch of kKernel with up to `bytes` of dynamic shared memory on the
// current device. The attribute belongs to the kernel on one device: it is set
// on the first launch there (threads that race for it set the same value).
template <auto kKernel>
[[nodiscard]] cudaError_t allow_smem(size_t bytes) {
    static std::atomic<uint64_t> allowed{0};  // bit d: device d; devices from 64 on are set each time
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const uint64_t bit = device < 64 ? uint64_t(1) << device : 0;
    if (allowed.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kKernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(bytes));
    if (e == cudaSuccess) allowed.fetch_or(bit, std::memory_order_release);
    return e;
}

} // namespace bj
