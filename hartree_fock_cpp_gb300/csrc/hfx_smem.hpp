// hfx_smem.hpp -- the dynamic shared-memory limit of a kernel.  The limit is
// an attribute of the kernel on one device: each device's own is raised, once,
// so that launches of concurrent jobs never race on it.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

namespace hfx {

// Runs raise() once per (device, kernel); after a failure the next call tries
// again.
class OncePerDevice {
public:
    template <typename F>
    cudaError_t run(int device, const void* kernel, F&& raise)
    {
        std::lock_guard<std::mutex> lk(mu_);
        if (done_.count({device, kernel})) return cudaSuccess;
        const cudaError_t e = raise();
        if (e == cudaSuccess) done_.insert({device, kernel});
        return e;
    }

private:
    std::mutex mu_;
    std::set<std::pair<int, const void*>> done_;
};

// The limit of `kernel` on the current device, raised to the device's maximum
// (hfx_kernels.cu).
cudaError_t allow_max_smem(const void* kernel);

}  // namespace hfx
