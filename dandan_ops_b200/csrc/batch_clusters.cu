// The batch kernel's clusters.
#include "batch_launch.cuh"

namespace b2host {

int launch_batch_clusters(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s) {
    if (p.deep) return launch_known<16, b2::kDeep>(xmap, a, p.grid, steps, overlap, s);
    return launch_rows<b2::kClusters>(p, xmap, a, steps, overlap, s);
}

}  // namespace b2host
