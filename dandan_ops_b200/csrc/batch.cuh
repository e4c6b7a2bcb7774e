// Host side of the batch kernel (batch.cu): its launch plan and the launch.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "batch_kernel.cuh"

namespace b2host {

struct BatchPlan {
    int nx;                // rows of x the accumulator holds: 16, 32, 64 or 128
    int row_tiles;         // more than one above 128 rows of x
    int steps;             // 64-column steps of all tiles
    int cluster;           // CTAs of a cluster, which share a tile; 1: ranges or rounds (or, deep, a cluster of one)
    bool deep;             // clusters with sixteen chains of products
    int whole;             // tiles that every CTA takes by itself; 0: equal ranges of steps
    int shared_tiles;      // the others, and the CTAs of each (rounds)
    int parts;
    int grid;
    int max_parts;         // most CTAs that share a tile
    int64_t partial_bytes;
};

// Partial tiles of any batch of up to m rows (more than 128 count as 128): grows with m, so a workspace that was sized for
// one batch holds the plan of every smaller one.  At most 19.4 MB.
inline int64_t batch_workspace(int64_t m, const b2::Dims& d, int sm_count) {
    const int64_t steps = int64_t((d.n + b2::kBatchRows - 1) / b2::kBatchRows) * d.kb * 4, sms = sm_count > 0 ? sm_count : 148;
    return b2::batch_partial_bytes(b2::batch_nx(m), int(steps < sms ? steps : sms));
}

BatchPlan plan_batch(int64_t m, const b2::Dims& d, int sm_count);
int launch_batch_ranges(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s);
int launch_batch_clusters(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s);
int launch_batch_rounds(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s);
int launch_batch_row_tiles(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s);
int launch_batch(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s);

}  // namespace b2host
