// Launch plan and launch of the batch kernel (batch_kernel.cuh).
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>

#include "../../include/b2_w4a16.h"
#include "batch.cuh"
#include "host_common.cuh"

namespace {

// Estimated time of a launch beyond its fixed start, in ns: the longest range of steps, the shared tiles in it (store, fence and
// ticket of each), and the reading of a tile's partial sums by the last CTA (measured on per-CTA time stamps).
int launch_cost(int nx, int steps, int tsteps, int grid) {
    const int range = (steps + grid - 1) / grid;
    const int tiles = steps / tsteps;
    const bool aligned = grid % tiles == 0;                     // every CTA inside one tile
    const int parts = aligned ? grid / tiles : (tsteps + range - 1) / range + 1;
    const int step_ns = nx <= 32 ? 220 : nx == 64 ? 250 : 310;
    return range * step_ns + (parts == 1 ? 0 : (aligned ? 1 : 2) * 1300 + parts * (200 + 7 * nx));
}

constexpr int kMaxPerTile = 16;      // CTAs per tile looked at: beyond, the partial sums cost more than the shorter ranges give

template <int NX, int STEPS>
int launch_one(const CUtensorMap& xmap, const b2::BatchArgs& a, int grid, bool overlap, cudaStream_t s) {
    auto kernel = b2::w4a16_batch_kernel<NX, STEPS>;
    constexpr int smem = b2::batch_smem_bytes(NX);
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return b2host::fail(B2_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
        configured.fetch_or(bit, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(b2::kBatchThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, xmap, a);
    if (e != cudaSuccess) return b2host::fail(B2_ERR_CUDA, std::string("w4a16_batch_kernel: ") + cudaGetErrorString(e));
    return b2host::after_launch("w4a16_batch_kernel");
}

}  // namespace

namespace b2host {

BatchPlan plan_batch(int64_t m, const b2::Dims& d, int sm_count) {
    BatchPlan p;
    p.nx = b2::batch_nx(m);
    const int tiles = (d.n + b2::kBatchRows - 1) / b2::kBatchRows, tsteps = d.kb * 4;
    const int64_t steps = int64_t(tiles) * tsteps;
    p.steps = int(steps);
    // Either equal ranges over all SMs, or the same number of CTAs for every tile (shorter hand-over, a few SMs idle):
    // 4096 x 4096 at M = 16 / 64: 148 CTAs 9.1 / 13.0 us, 4 per tile 7.3 / 10.9; 1024 x 2048 at M = 32: 85 CTAs 7.9 us, 24 CTAs 5.8.
    const int sms = int(std::min<int64_t>(sm_count > 0 ? sm_count : 148, steps));
    int best_cost = launch_cost(p.nx, p.steps, tsteps, sms);
    p.grid = sms;
    for (int g = tiles; g <= std::min(sms, kMaxPerTile * tiles); g += tiles) {
        const int cost = launch_cost(p.nx, p.steps, tsteps, g);
        if (cost <= best_cost) { best_cost = cost; p.grid = g; }
    }
    const int64_t range = (steps + p.grid - 1) / p.grid;
    p.max_parts = p.grid % tiles == 0 ? p.grid / tiles : int(std::min<int64_t>(p.grid, (tsteps + range - 1) / range + 1));
    p.partial_bytes = b2::batch_partial_bytes(p.nx, p.grid);
    return p;
}

template <int NX>
int launch_known(const CUtensorMap& xmap, const b2::BatchArgs& a, int grid, int steps, bool overlap, cudaStream_t s) {
    if (steps == b2::kStepsFp16) return launch_one<NX, b2::kStepsFp16>(xmap, a, grid, overlap, s);
    if (steps == b2::kStepsPlain) return launch_one<NX, b2::kStepsPlain>(xmap, a, grid, overlap, s);
    return launch_one<NX, b2::kStepsMixed>(xmap, a, grid, overlap, s);
}

int launch_batch(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s) {
    switch (p.nx) {
        case 16: return launch_known<16>(xmap, a, p.grid, steps, overlap, s);
        case 32: return launch_known<32>(xmap, a, p.grid, steps, overlap, s);
        case 64: return launch_known<64>(xmap, a, p.grid, steps, overlap, s);
        default: return launch_known<128>(xmap, a, p.grid, steps, overlap, s);
    }
}

}  // namespace b2host
