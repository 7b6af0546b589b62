// Opt-in of a kernel to more than 48 KB of dynamic shared memory.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace rsgpu {

// The limit belongs to a kernel on one device, and a process may hold plans on several:
// raised once on each device that launches the kernel, at any number of threads.  Later
// launches cost a cudaGetDevice and an atomic load.
class SmemLimit {
public:
    template <typename... P>
    cudaError_t raise(void (*kernel)(P...), size_t bytes)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const unsigned long long bit = dev < 64 ? 1ull << dev : 0;   // beyond: raised at each launch
        if (raised.load(std::memory_order_acquire) & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(reinterpret_cast<const void *>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) raised.fetch_or(bit, std::memory_order_release);
        return e;
    }

private:
    std::atomic<unsigned long long> raised{0};
};

}  // namespace rsgpu
