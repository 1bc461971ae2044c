// pf3d_once.h -- set-up that a kernel needs once on every device it is
// launched on (its shared-memory limit is an attribute per device).
#pragma once
#include <cuda_runtime.h>
#include <atomic>

namespace pf3d {

struct DeviceOnce {
    std::atomic<unsigned long long> done{0};   // devices set up, a bit each; those beyond 63 are set up at each call
    template <typename F>
    cudaError_t operator()(F set_up)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
        if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
        e = set_up();
        if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

}  // namespace pf3d
