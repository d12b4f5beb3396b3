// Host side of the cluster solvers: launch configuration and how many clusters of a
// shape are resident at once.
#pragma once

#include <map>
#include <mutex>
#include <tuple>

#include <cuda_runtime.h>

namespace dwfb {

struct ClusterLaunch
{
    int CS = 0, R = 0;  // CTAs per cluster, time rows per CTA
    int NL = 0, LT = 0;  // threads per site, slices per thread
    int threads = 0, resident = 0;
    size_t smem = 0;
    const void* fn = nullptr;

    void config(int clusters, cudaStream_t stream, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr) const
    {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = unsigned(CS);
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg = cudaLaunchConfig_t{};
        cfg.gridDim = dim3(unsigned(CS * clusters));
        cfg.blockDim = dim3(unsigned(threads));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

// Clusters of this shape resident at once on the device (0: none; kernel attributes,
// shared memory up to smem_max, set on the way), queried once per device and shape, so
// that a later call, the one a stream capture records, issues the launch alone. A
// failed query counts as none for this call only and takes no error away that was
// pending before it.
inline int resident_clusters(const ClusterLaunch& s, int device, size_t smem_max)
{
    using Key = std::tuple<int, const void*, int, int, size_t>;
    static std::map<Key, int> known;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    const Key key(device, s.fn, s.CS, s.threads, s.smem);
    const auto it = known.find(key);
    if (it != known.end())
        return it->second;
    const bool clean = cudaPeekAtLastError() == cudaSuccess;
    int n = 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    s.config(1, nullptr, cfg, attr);
    if (cudaFuncSetAttribute(s.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_max)) != cudaSuccess ||
        cudaFuncSetAttribute(s.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, s.fn, &cfg) != cudaSuccess)
    {
        if (clean)
            cudaGetLastError();
        return 0;
    }
    known[key] = n;
    return n;
}

}  // namespace dwfb
