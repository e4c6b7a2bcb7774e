// Residual add + RMSNorm of one row, shared by the standalone norm kernel and the tile kernel's fused
// prologue, so that both produce the same bits.  Rounding order of the reference
// (dandan_ops/csrc/elementwise.cu:39-62, dandan_ops/elementwise.py:118-120): the sum is rounded to FP16
// first, the normalized value is rounded to FP16 before the weight multiplies it.
#pragma once
#include "stream_kernel.cuh"

namespace b2 {

constexpr int kNormThreads = 32 * kNormSlices;       // the first 256 threads of the CTA do the work

struct NormScratch {                                   // shared memory of one row's reduction
    float slice[kNormSlices];
};

// One row: summed = fp16(x + residual) (to `sums`: the caller's `summed` row, or the output row when the sum is
// not wanted), out = fp16(fp16(s * inverse_rms(s)) * weight).  Every thread of the CTA must call it (it
// contains a block-wide barrier); threads beyond kNormThreads only take part in that.  The sum of
// squares is added in eight lane-strided slices (one per warp), butterfly inside a slice, slices in order: a
// fixed order, so the result does not depend on the launch.
__device__ __forceinline__ void norm_row(const __half* x, const __half* residual, const __half* weight, float eps,
                                         __half* sums, __half* out, int k, NormScratch& sm) {
    const int pieces = k >> 3;
    constexpr int kStride = kNormThreads, kBatch = 4;  // loads in flight per thread; the sum keeps the order of the pieces
    const bool worker = threadIdx.x < kNormThreads;
    // Up to 8192 columns a thread keeps its pieces of the sum (and has requested their weights) until the mean is known; longer
    // rows are read back.  x and residual through L2: as a programmatic dependent the kernel is older than what the previous
    // one has written.
    const bool held = pieces <= kStride * kBatch;
    uint4 v[kBatch], w[kBatch];
    float sq = 0.0f;
    if (worker) {
        for (int c0 = threadIdx.x; c0 < pieces; c0 += kStride * kBatch) {
            uint4 r[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int cc = c0 + kStride * j;
                v[j] = cc < pieces ? __ldcg(reinterpret_cast<const uint4*>(x + cc * 8)) : make_uint4(0, 0, 0, 0);
                r[j] = (cc < pieces && residual) ? __ldcg(reinterpret_cast<const uint4*>(residual + cc * 8)) : make_uint4(0, 0, 0, 0);
                if (held && cc < pieces) w[j] = __ldcg(reinterpret_cast<const uint4*>(weight + cc * 8));
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int cc = c0 + kStride * j;
                if (cc < pieces) {
                    if (residual) v[j] = add_piece(v[j], r[j]);
                    if (!held || sums != out) *reinterpret_cast<uint4*>(sums + cc * 8) = v[j];
                    sq = sumsq_piece(v[j], sq);
                }
            }
        }
        sq = warp_sum(sq);
        if ((threadIdx.x & 31) == 0) sm.slice[threadIdx.x >> 5] = sq;
    }
    __syncthreads();
    float total = 0.0f;                                // (every thread for itself: no second barrier)
#pragma unroll
    for (int p = 0; p < kNormSlices; ++p) total += sm.slice[p];
    const float inverse = inverse_rms(total, k, eps);
    if (worker) {
        for (int c0 = threadIdx.x; c0 < pieces; c0 += kStride * kBatch) {      // every thread re-reads only what it wrote itself
            if (!held) {
#pragma unroll
                for (int j = 0; j < kBatch; ++j) {
                    const int cc = c0 + kStride * j;
                    if (cc < pieces) {
                        v[j] = *reinterpret_cast<const uint4*>(sums + cc * 8);
                        w[j] = __ldcg(reinterpret_cast<const uint4*>(weight + cc * 8));
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int cc = c0 + kStride * j;
                if (cc < pieces) *reinterpret_cast<uint4*>(out + cc * 8) = norm_piece(v[j], inverse, w[j]);
            }
        }
    }
}

}  // namespace b2
