// Launch helpers shared by the step kernels' translation units.
#pragma once

#include "cheb_kernels.cuh"

#include <mutex>
#include <unordered_map>

namespace rsatb_b200 {
namespace step_detail {

constexpr int kNotApplicable = 1000;

// Resident CTAs per SM for a kernel at a given CTA size and shared memory.
inline int occupancy(const void* kernel, int threads, size_t smem) {
    static std::mutex mu;
    static std::unordered_map<uint64_t, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t key = (uint64_t(reinterpret_cast<uintptr_t>(kernel)) << 8) ^
                         (uint64_t(threads) << 40) ^ (uint64_t(smem) << 20) ^ uint64_t(dev);
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    int n = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess ||
        n < 1)
        n = 1;
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = n;
    return n;
}

// The any-shape FP64 tensor-core kernel (cheb_dmma_any_f64.cu, _f32.cu): blocks
// of 2 to 8, widths up to 256 reals; kNotApplicable otherwise.
template <typename VT, bool CM, bool CV>
int launch_dmma_any(rsatb_context* ctx, StepArgs& a);

}  // namespace step_detail
}  // namespace rsatb_b200
