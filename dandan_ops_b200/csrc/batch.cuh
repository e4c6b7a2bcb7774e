// Host side of the batch kernel (batch.cu): its launch plan and the launch.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "batch_kernel.cuh"

namespace b2host {

struct BatchPlan {
    int nx;                // rows of x the accumulator holds: 16, 32, 64 or 128
    int steps;             // 64-column steps of all tiles
    int grid;
    int max_parts;         // most CTAs that share a tile
    int64_t partial_bytes;
};

BatchPlan plan_batch(int64_t m, const b2::Dims& d, int sm_count);
int launch_batch(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, bool h16, bool overlap, cudaStream_t s);

}  // namespace b2host
