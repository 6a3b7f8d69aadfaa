// How thread-block clusters of a kernel pack into the current device.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>

namespace opsnn {

// How many clusters of s CTAs of `kernel` the current device keeps resident at once under a cluster scheduling policy
// (cudaClusterSchedulingPolicy*: 0 default / 1 spread / 2 load balancing). Answers are cached per (kernel, device, s, policy).
inline int max_active_clusters(const void* kernel, int threads, int smem_bytes, int s, int policy)
{
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, int, int>, int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(kernel, dev, s, policy);
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(s * 64), 1, 1);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeClusterSchedulingPolicyPreference;
    attr[1].val.clusterSchedulingPolicyPreference = static_cast<cudaClusterSchedulingPolicy>(policy);
    cfg.attrs = attr;
    cfg.numAttrs = policy != 0 ? 2 : 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = n;
    return n;
}

// Largest cluster size S in [2, max_s] for which `clusters` clusters of S CTAs of `kernel` are all resident at once on the
// current device (default scheduling policy), 0 when there is none.
inline int pick_cluster_size(const void* kernel, int threads, int smem_bytes, int64_t clusters, int max_s)
{
    for (int s = max_s; s >= 2; --s)
        if ((int64_t)max_active_clusters(kernel, threads, smem_bytes, s, 0) >= clusters) return s;
    return 0;
}

}  // namespace opsnn
