// Resident blocks per SM of the library's kernels.
#include <map>
#include <mutex>
#include <tuple>

#include "internal.hpp"

namespace tgtp {

// The dynamic shared-memory limit is an attribute of the kernel on one device, so the record of the
// limits raised so far is kept per device, like the results.
int blocks_per_sm(const void* kern, int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, size_t, int>, int> cache;
    static std::map<std::pair<const void*, int>, size_t> limit;
    int dev = 0;
    TGTP_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(kern, threads, smem, dev);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    size_t& most = limit[{kern, dev}];
    if (smem > most) {
        TGTP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        most = smem;
    }
    int per_sm = 0;
    TGTP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    cache[key] = per_sm;
    return per_sm;
}

}  // namespace tgtp
