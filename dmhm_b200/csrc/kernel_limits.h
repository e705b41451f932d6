// Per-device attributes of kernels: the dynamic shared memory a kernel may use
// and how many of its CTAs an SM holds.  A process may have contexts on several
// devices, and both belong to one device's copy of a kernel, so they are kept
// by (device, kernel); contexts on several host threads may ask at once.
#pragma once
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

#include "common.h"

namespace hmb {

// The largest value recorded per (device, kernel).
class KernelRecord {
  public:
    // Runs set() unless at least `bytes` are recorded; records them if it returns.
    template <typename F>
    void raise(int device, const void* kernel, size_t bytes, F set) {
        std::lock_guard<std::mutex> lock(mu_);
        auto f = have_.find({device, kernel});
        if (f != have_.end() && f->second >= bytes) return;
        set();
        have_[{device, kernel}] = bytes;
    }
    // The recorded value, or what find() returns, recorded.
    template <typename F>
    size_t get(int device, const void* kernel, F find) {
        std::lock_guard<std::mutex> lock(mu_);
        auto f = have_.find({device, kernel});
        if (f != have_.end()) return f->second;
        const size_t v = find();
        have_[{device, kernel}] = v;
        return v;
    }

  private:
    std::mutex mu_;
    std::map<std::pair<int, const void*>, size_t> have_;
};

inline int current_device() {
    int dev = 0;
    HMB_CUDA(cudaGetDevice(&dev));
    return dev;
}

#ifdef __CUDACC__
// Lets launches of `kernel` on the current device use `bytes` of dynamic shared memory.
template <typename K>
void allow_smem(K kernel, size_t bytes) {
    static KernelRecord done;
    const void* k = reinterpret_cast<const void*>(kernel);
    done.raise(current_device(), k, bytes, [&] {
        HMB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    });
}

// CTAs of `kernel` (always launched with these threads and shared memory) that
// an SM of the current device holds.
template <typename K>
int ctas_per_sm(K kernel, int threads, size_t smem = 0) {
    static KernelRecord found;
    const void* k = reinterpret_cast<const void*>(kernel);
    return (int)found.get(current_device(), k, [&] {
        int n = 0;
        HMB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, smem));
        return (size_t)std::max(1, n);
    });
}
#endif

}  // namespace hmb
