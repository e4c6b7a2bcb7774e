// Plain step fields of a native image -> factored ones where that gives the same weights (layout.cuh).
#pragma once
#include "layout.cuh"

namespace b2 {

constexpr int kFactorSet = 16;                                  // candidates for a1 of which the best is checked
struct FactorTable { float inverse[128]; };                     // 128 / (128 + i)
constexpr FactorTable factor_table() {
    FactorTable t = {};
    for (int i = 0; i < 128; ++i) t.inverse[i] = 128.0f / float(128 + i);
    return t;
}
__constant__ constexpr FactorTable kFactorTable = factor_table();

// The fields of eight blocks per CTA.  With m the mantissa of a step (1 <= m < 2), t = m / a1 is rounded to a multiple of 2^-10 (by
// adding and subtracting 1.5 * 2^13) and the distance m - a1 * a2 is exact in one fma: no conversions, the same candidates
// in all lanes.  The best of sixteen candidates has a remainder of about 2^-16 and reproduces all weights in six of seven
// cases, which is then checked with the very operations the kernels decode with; the steps that are left are closed up
// and looked at with the next sixteen candidates.  A step that a1 = 1 gives without a remainder is found in the
// first set (its key is the smallest there is).
//
// A field changes from one valid form to the other in one 4-byte store, so a kernel that reads the image meanwhile decodes the
// same weights.
constexpr int kFactorThreads = 512, kFactorBlocks = kFactorThreads / 64;
__global__ void __launch_bounds__(kFactorThreads)
factor_steps_kernel(uint8_t* native, int64_t blocks) {
    __shared__ float steps[kFactorThreads];
    __shared__ uint8_t zeros[kFactorThreads];
    __shared__ uint16_t list[2][kFactorThreads];
    __shared__ int count[2];
    __shared__ float inverses[128];                                          // (constant memory answers one address at a time)
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t block0 = int64_t(blockIdx.x) * kFactorBlocks;
    if (tid < 2) count[tid] = 0;
    if (tid < 128) inverses[tid] = 128.0f / float(128 + tid);
    __syncthreads();
    auto append = [&](int which, int entry, bool yes) {                      // (called by whole warps)
        const unsigned votes = __ballot_sync(0xffffffffu, yes);
        int at = 0;
        if (lane == 0 && votes) at = atomicAdd(&count[which], __popc(votes));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (yes) list[which][at + __popc(votes & ((1u << lane) - 1u))] = uint16_t(entry);
    };
    {
        const int64_t block = block0 + (tid >> 6);
        const int f = tid & 63;
        float s = 0.0f;
        if (block < blocks) {
            const uint8_t* base = native + block * kBlockBytes;
            const uint32_t field = reinterpret_cast<const uint32_t*>(base + kStepOffset)[f];
            s = int32_t(field) < 0 ? 0.0f : __uint_as_float(field);
            zeros[tid] = (base[kZeroOffset + (f >> 1)] >> (4 * (f & 1))) & 15u;
        }
        steps[tid] = s;
        append(0, tid, s >= 0x1p-12f && s < 3.99f);
    }
    constexpr float kMagic = 12288.0f;
    for (int set = 0, cur = 0; set < 128; set += kFactorSet, cur ^= 1) {
        __syncthreads();
        const int todo = count[cur];
        if (todo == 0) break;
        if ((tid & ~31) < todo) {
            const bool active = tid < todo;
            const int entry = list[cur][active ? tid : 0];
            const float s = steps[entry];
            const uint32_t z = zeros[entry], bits = __float_as_uint(s);
            const float m = __uint_as_float((bits & 0x007FFFFFu) | 0x3F800000u);
            const float scale = __uint_as_float(bits & 0x7F800000u);         // s = m * scale
            const float base = -1.0f - float(set) * 0x1p-7f;
            unsigned best = 0xffffffffu;                                     // |distance| with the candidate's number in the low bits
#pragma unroll
            for (int i = 0; i < kFactorSet; i += 2) {
                float d0, d1;
                const float2 inverse = make_float2(kFactorTable.inverse[set + i], kFactorTable.inverse[set + i + 1]);
                const float a0 = base - float(i) * 0x1p-7f, a1 = base - float(i + 1) * 0x1p-7f;
                asm("{\n\t.reg .b64 t, m, c, a;\n\t"
                    "mov.b64 m, {%2, %2};\n\tmov.b64 t, {%3, %4};\n\tmov.b64 c, {%5, %5};\n\tmov.b64 a, {%6, %7};\n\t"
                    "mul.rn.f32x2 t, m, t;\n\tadd.rn.f32x2 t, t, c;\n\tsub.rn.f32x2 t, t, c;\n\tfma.rn.f32x2 t, a, t, m;\n\t"
                    "mov.b64 {%0, %1}, t;\n\t}"
                    : "=f"(d0), "=f"(d1) : "f"(m), "f"(inverse.x), "f"(inverse.y), "f"(kMagic), "f"(a0), "f"(a1));
                best = min(best, min((__float_as_uint(d0) & 0x7FFFFFF0u) | unsigned(i), (__float_as_uint(d1) & 0x7FFFFFF0u) | unsigned(i + 1)));
            }
            const int i = set + int(best & 15u);
            const float a1 = 1.0f + float(i) * 0x1p-7f;
            const float a2 = __fsub_rn(__fadd_rn(__fmul_rn(m, inverses[i]), kMagic), kMagic);
            const int remainder = int(bits) - __float_as_int(a1 * a2 * scale);
            const uint32_t a2_bits = __half_as_ushort(__float2half_rn(a2 * scale * 0x1p14f));
            const __half2 a2_pair = __half2half2(__ushort_as_half(uint16_t(a2_bits)));
            const __half2 even = __half2half2(__ushort_as_half(uint16_t(0x6400u | unsigned(i) << 3)));      // a1 * 2^10
            const __half2 b = __hmul2(even, __half2half2(__ushort_as_half(uint16_t(0x8000u | z))));         // -z * a1 * 2^-14
            uint32_t differ = unsigned(remainder + 512) < 1024u ? 0u : 1u;
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
                const float d = float(c) - float(z);
                const __half2 want = __floats2half2_rn(__fmul_rn(d, s), __fmul_rn(d + 1.0f, s));
                const uint32_t codes = uint32_t(c) | uint32_t(c + 1) << 16;   // as FP16: code * 2^-24
                const __half2 got = __hmul2(__hfma2(*reinterpret_cast<const __half2*>(&codes), even, b), a2_pair);
                differ |= *reinterpret_cast<const uint32_t*>(&got) ^ *reinterpret_cast<const uint32_t*>(&want);
            }
            if (active && differ == 0)
                reinterpret_cast<uint32_t*>(native + (block0 + (entry >> 6)) * kBlockBytes + kStepOffset)[entry & 63] =
                    factored_field(uint32_t(i), a2_bits, remainder);
            append(cur ^ 1, entry, active && differ != 0);
        }
        __syncthreads();
        if (tid == 0) count[cur] = 0;
    }
}

}  // namespace b2
