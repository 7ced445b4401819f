// Blocks of a kernel that the current device holds at once (SMs x blocks per
// SM), asked of the runtime once per device and kernel.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace cfs {

struct ResidentCache {
    static constexpr int kMaxDev = 64;
    std::once_flag once[kMaxDev];
    long long blocks[kMaxDev] = {};
};

// 0 when the query fails (no error is left behind).
template <class Kernel>
long long resident_blocks(ResidentCache& cache, Kernel kernel, int threads, size_t dyn) {
    auto query = [&](int dev) -> long long {
        int per_sm = 0, sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, dyn) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
        return static_cast<long long>(per_sm) * sms;
    };
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    if (dev < 0 || dev >= ResidentCache::kMaxDev) return query(dev);
    std::call_once(cache.once[dev], [&] { cache.blocks[dev] = query(dev); });
    return cache.blocks[dev];
}

}  // namespace cfs
