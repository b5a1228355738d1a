// grid_cache.h -- grid sizes of the persistent kernels, and the stack words they are kept by.
#pragma once
#include <mutex>
#include <cuda_runtime_api.h>

namespace timrt {

constexpr int kStackSize = 32;   // the reference's bitstack is 32 bits wide
// Most stack words of a thread of k_walk (walk.cuh): a closest-hit ray of the binary form
// leaves one child a level waiting, a ray of the 8-wide form two words a level (kernels.h:
// has_walk), and both have an end marker and the word above the top. And the most words
// that a thread keeps beside its stack (walk_words).
constexpr int kWalkStack = kStackSize + 2, kWalkBeside = 12;

// Grid sizes of one persistent kernel, per device ordinal and stack depth: the
// occupancy calculator's resident blocks per SM times the device's SM count,
// computed on first use with the device current (which also sets the kernel's
// dynamic shared-memory limit in that device's context). Thread-safe.
struct GridCache {
    static constexpr int kDevices = 64, kDepths = kWalkStack + kWalkBeside + 1;   // depths 0 and up
    std::mutex mu;
    int blocks[kDevices][kDepths] = {};
    template <class F>
    int get(int depth, F compute) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) {
            cudaGetLastError();
            dev = -1;
        }
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0) return compute(0);
        if (depth < 0 || depth >= kDepths) return compute(dev);   // no launcher asks for one
        if (!blocks[dev][depth]) blocks[dev][depth] = compute(dev);
        return blocks[dev][depth];
    }
};

}  // namespace timrt
