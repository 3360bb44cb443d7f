// What a launcher asks or sets once per GPU.  A process may drive several GPUs: launch attributes hold for the device that is
// current when they are set, and devices need not have the same number of SMs.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include "hccl/hccl_types.h"

namespace hccl {

constexpr int kMaxDevices = 64;

// Runs `set` (returning HcclResult) until it has succeeded once on the current device.  On a device that cannot be named
// it runs every time.
class OncePerDevice {
public:
    template <class F>
    HcclResult operator()(F&& set)
    {
        int dev = -1;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return set();
        if (done_[dev].load(std::memory_order_acquire)) return HCCL_SUCCESS;
        const HcclResult r = set();
        if (r == HCCL_SUCCESS) done_[dev].store(true, std::memory_order_release);
        return r;
    }

private:
    std::atomic<bool> done_[kMaxDevices] = {};
};

// SMs of the current device; those of a B200 where it cannot be asked.
inline int SmCount()
{
    static std::atomic<int> count[kMaxDevices] = {};
    int dev = -1, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 148;
    if (dev < kMaxDevices && (n = count[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 148;
    if (dev < kMaxDevices) count[dev].store(n, std::memory_order_relaxed);
    return n;
}

}  // namespace hccl
