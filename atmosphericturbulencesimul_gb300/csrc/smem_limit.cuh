// smem_limit.cuh -- a kernel's dynamic shared memory above the default.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <atomic>

namespace atmwfs {

// Raises one kernel's limit before its first launch on each device.  The limit
// belongs to the kernel on the current device, so the record is one bit per
// device (the first 64; beyond, and where several threads make a first launch,
// it is set again, which changes nothing).
class SmemLimit {
public:
    template <typename K>
    cudaError_t raise(K kern, size_t bytes)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
        if (done_.load(std::memory_order_relaxed) & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kern), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_relaxed);
        return e;
    }

private:
    std::atomic<unsigned long long> done_{0};
};

}  // namespace atmwfs
