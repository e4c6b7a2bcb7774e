// Launches of the batch kernel, for the translation units that hold its forms (a unit per form: a program loads those it uses).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <string>

#include "../../include/b2_w4a16.h"
#include "batch.cuh"
#include "host_common.cuh"

namespace b2host {
namespace {                       // (what is configured is known per copy of the library: no symbol shared between two of them)

template <int NX, int STEPS, int FORM, bool MANY>
int launch_one(const CUtensorMap& xmap, const b2::BatchArgs& a, int grid, bool overlap, cudaStream_t s) {
    auto kernel = b2::w4a16_batch_kernel<NX, STEPS, FORM, MANY>;
    constexpr bool CL = FORM == b2::kClusters || FORM == b2::kDeep;
    constexpr int smem = b2::batch_smem_bytes(NX, FORM);
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail(B2_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
        configured.fetch_or(bit, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(b2::kBatchThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int count = 0;
    if (CL) {
        attr[count].id = cudaLaunchAttributeClusterDimension;
        attr[count].val.clusterDim.x = unsigned(a.cluster); attr[count].val.clusterDim.y = 1; attr[count].val.clusterDim.z = 1;
        ++count;
    }
    if (overlap) {
        attr[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[count].val.programmaticStreamSerializationAllowed = 1;
        ++count;
    }
    cfg.attrs = attr;
    cfg.numAttrs = unsigned(count);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, xmap, a);
    if (e != cudaSuccess) return fail(B2_ERR_CUDA, std::string("w4a16_batch_kernel: ") + cudaGetErrorString(e));
    return after_launch("w4a16_batch_kernel");
}

template <int NX, int FORM, bool MANY = false>
int launch_known(const CUtensorMap& xmap, const b2::BatchArgs& a, int grid, int steps, bool overlap, cudaStream_t s) {
    if (steps == b2::kStepsFp16) return launch_one<NX, b2::kStepsFp16, FORM, MANY>(xmap, a, grid, overlap, s);
    if (steps == b2::kStepsPlain) return launch_one<NX, b2::kStepsPlain, FORM, MANY>(xmap, a, grid, overlap, s);
    return launch_one<NX, b2::kStepsMixed, FORM, MANY>(xmap, a, grid, overlap, s);
}

template <int FORM>
int launch_rows(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s) {
    switch (p.nx) {
        case 16: return launch_known<16, FORM>(xmap, a, p.grid, steps, overlap, s);
        case 32: return launch_known<32, FORM>(xmap, a, p.grid, steps, overlap, s);
        case 64: return launch_known<64, FORM>(xmap, a, p.grid, steps, overlap, s);
        default: return launch_known<128, FORM>(xmap, a, p.grid, steps, overlap, s);
    }
}

}  // namespace
}  // namespace b2host
