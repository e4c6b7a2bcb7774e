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

// A thread takes one field.  With m the mantissa of its step (1 <= m < 2), t = m / a1 is rounded to a multiple of 2^-10 (by adding
// and subtracting 1.5 * 2^13) and the distance m - a1 * a2 is exact in one fma: no conversions, the same candidates in all
// lanes.  The best of sixteen candidates has a remainder of about 2^-16 and reproduces all weights in six of seven cases, which is
// then checked with the very operations the kernels decode with; a warp needs 2.6 such sets on average.  A step that a1 = 1
// gives without a remainder is found in the first set (its key is the smallest there is).
//
// A field changes from one valid form to the other in one 4-byte store, so a kernel that reads the image meanwhile decodes the
// same weights.  Measured on 4096 x 12288 (786432 steps): see b2_w4a16_factor_steps().
__global__ void __launch_bounds__(256)
factor_steps_kernel(uint8_t* native, int64_t blocks) {
    const int64_t index = int64_t(blockIdx.x) * 256 + threadIdx.x, block = index >> 6;
    const int f = int(index & 63);
    uint32_t* at = nullptr;
    float s = 0.0f;
    uint32_t z = 0;
    if (block < blocks) {
        uint8_t* base = native + block * kBlockBytes;
        at = reinterpret_cast<uint32_t*>(base + kStepOffset) + f;
        const uint32_t field = *at;
        s = int32_t(field) < 0 ? 0.0f : __uint_as_float(field);
        z = (base[kZeroOffset + (f >> 1)] >> (4 * (f & 1))) & 15u;
    }
    bool open = s >= 0x1p-12f && s < 3.99f;
    const uint32_t bits = __float_as_uint(s);
    const float m = __uint_as_float((bits & 0x007FFFFFu) | 0x3F800000u);
    const float scale = __uint_as_float(bits & 0x7F800000u);                 // s = m * scale
    constexpr float kMagic = 12288.0f;
    for (int set = 0; set < 128 && __any_sync(0xffffffffu, open); set += kFactorSet) {
        unsigned best = 0xffffffffu;                                         // |distance| with the candidate's number in the low bits
#pragma unroll
        for (int i = 0; i < kFactorSet; i += 2) {
            float d0, d1;
            const float2 inverse = make_float2(kFactorTable.inverse[set + i], kFactorTable.inverse[set + i + 1]);
            const float a0 = -(1.0f + float(set + i) * 0x1p-7f), a1 = a0 - 0x1p-7f;
            asm("{\n\t.reg .b64 t, m, c, a;\n\t"
                "mov.b64 m, {%2, %2};\n\tmov.b64 t, {%3, %4};\n\tmov.b64 c, {%5, %5};\n\tmov.b64 a, {%6, %7};\n\t"
                "mul.rn.f32x2 t, m, t;\n\tadd.rn.f32x2 t, t, c;\n\tsub.rn.f32x2 t, t, c;\n\tfma.rn.f32x2 t, a, t, m;\n\t"
                "mov.b64 {%0, %1}, t;\n\t}"
                : "=f"(d0), "=f"(d1) : "f"(m), "f"(inverse.x), "f"(inverse.y), "f"(kMagic), "f"(a0), "f"(a1));
            best = min(best, min((__float_as_uint(d0) & 0x7FFFFFF0u) | unsigned(i), (__float_as_uint(d1) & 0x7FFFFFF0u) | unsigned(i + 1)));
        }
        const int i = set + int(best & 15u);
        const float a1 = 1.0f + float(i) * 0x1p-7f;
        const float a2 = __fsub_rn(__fadd_rn(__fmul_rn(m, kFactorTable.inverse[i]), kMagic), kMagic);
        const int remainder = int(bits) - __float_as_int(a1 * a2 * scale);
        const uint32_t a2_bits = __half_as_ushort(__float2half_rn(a2 * scale * 0x1p14f));
        const __half2 a2_pair = __half2half2(__ushort_as_half(uint16_t(a2_bits)));
        const __half2 even = __half2half2(__ushort_as_half(uint16_t(0x6400u | unsigned(i) << 3)));          // a1 * 2^10
        const __half2 b = __hmul2(even, __half2half2(__ushort_as_half(uint16_t(0x8000u | z))));             // -z * a1 * 2^-14
        uint32_t differ = unsigned(remainder + 512) < 1024u ? 0u : 1u;
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
            const float d = float(c) - float(z);
            const __half2 want = __floats2half2_rn(__fmul_rn(d, s), __fmul_rn(d + 1.0f, s));
            const uint32_t codes = uint32_t(c) | uint32_t(c + 1) << 16;       // as FP16: code * 2^-24
            const __half2 got = __hmul2(__hfma2(*reinterpret_cast<const __half2*>(&codes), even, b), a2_pair);
            differ |= *reinterpret_cast<const uint32_t*>(&got) ^ *reinterpret_cast<const uint32_t*>(&want);
        }
        if (open && differ == 0) {
            *at = factored_field(uint32_t(i), a2_bits, remainder);
            open = false;
        }
    }
}

}  // namespace b2
