// The batch kernel's clusters.
#include "batch_launch.cuh"

namespace b2host {

// Clusters of c CTAs of the kernel that the device runs at the same time (asked once per device and size; without a device, for
// planning alone, those of a B200).
int cluster_capacity(int c) {
    static std::atomic<int> known[64][9];                    // 0 = not asked yet, else capacity + 1
    static constexpr int kB200[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return kB200[c];
    }
    std::atomic<int>& at = known[dev][c];
    if (const int v = at.load(std::memory_order_acquire)) return v - 1;
    auto kernel = b2::w4a16_batch_kernel<16, b2::kStepsMixed, b2::kClusters>;
    constexpr int smem = 232448;                             // (no form uses more)
    int clusters = 0;
    bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
    if (ok) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(unsigned(c));
        cfg.blockDim = dim3(b2::kBatchThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = unsigned(c); attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        ok = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();                                  // clear the error of a failed query
        clusters = 0;
    }
    at.store(clusters + 1, std::memory_order_release);
    return clusters;
}

int launch_batch_clusters(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s) {
    return launch_rows<b2::kClusters>(p, xmap, a, steps, overlap, s);
}

}  // namespace b2host
