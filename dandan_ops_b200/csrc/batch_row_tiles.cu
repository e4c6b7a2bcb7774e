// The batch kernel over more than 128 rows of x: clusters, or a tile per CTA.
#include "batch_launch.cuh"

namespace b2host {

int launch_batch_row_tiles(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s) {
    if (p.cluster > 1) return launch_known<128, b2::kClusters, true>(xmap, a, p.grid, steps, overlap, s);
    if (p.whole) return launch_known<128, b2::kRounds, true>(xmap, a, p.grid, steps, overlap, s);
    return fail(B2_ERR_UNSUPPORTED, "the batch kernel takes equal ranges up to 128 rows of x");
}

}  // namespace b2host
