// Plain step fields of a native image -> factored ones where that gives the same weights (layout.cuh).
#pragma once
#include "layout.cuh"

namespace b2 {

constexpr int kFactorWarps = 4, kFactorThreads = 32 * kFactorWarps;
constexpr int kFactorMaxBlocks = 8;                             // blocks of a warp
constexpr int kFactorSet = 16;                                  // candidates for a1 of which the nearest is checked
constexpr int kFactorShared = 3;                                // sets after which the CTA closes up what is left
constexpr int kFactorMisses = 16;                               // most steps outside the factored range in a block that is searched
struct FactorTable {
    float inverse[128];                                         // 128 / (128 + i)
    uint32_t scaled[128];                                       // 2^26 / (128 + i)
};
constexpr FactorTable factor_table() {
    FactorTable t = {};
    for (int i = 0; i < 128; ++i) {
        t.inverse[i] = 128.0f / float(128 + i);
        t.scaled[i] = ((1u << 27) / uint32_t(128 + i) + 1) / 2;
    }
    return t;
}
__constant__ constexpr FactorTable kFactorTable = factor_table();

// A step and what its candidates share: s = m * scale, 1 <= m < 2.
struct FactorStep {
    float s, m, scale;
    uint32_t z;
    __device__ __forceinline__ FactorStep(float step, uint32_t zero) : s(step), z(zero) {
        m = __uint_as_float((__float_as_uint(s) & 0x007FFFFFu) | 0x3F800000u);
        scale = __uint_as_float(__float_as_uint(s) & 0x7F800000u);
    }
    // a2 / (scale * 2^14) for a1 = 1 + i / 128: m / a1 rounded to the spacing that FP16 numbers have there (2^-11 below 1, else
    // 2^-10), by adding and subtracting 1.5 * 2^12 or 1.5 * 2^13
    __device__ __forceinline__ float magic(float a1) const { return m < a1 ? 6144.0f : 12288.0f; }
    __device__ __forceinline__ float a2(float inverse, float magic) const { return __fsub_rn(__fmaf_rn(m, inverse, magic), magic); }
    __device__ __forceinline__ int remainder(float a1, float a2) const { return __float_as_int(s) - __float_as_int(a1 * a2 * scale); }
};
__device__ __forceinline__ float factor_a1(uint32_t i) { return __uint_as_float(0x3F800000u + (i << 16)); }

// The field of a step if the nearest of the sixteen candidates from `set` on gives its weights, else 0.  `scaled(i)`: 2^26 / (128 +
// set + i).  m * 2^23 times that is m / a1 in units of 2^-42, so its low 32 bits, read with a sign, are the distance of m / a1 from the
// next multiple of 2^-10 (doubled: 2^-11): one integer multiplication per candidate.  Smallest and largest of them are the nearest on
// either side.
template <typename Scaled>
__device__ __forceinline__ uint32_t factor_nearest(const FactorStep& f, int set, const float* inverses, const uint2* masks, const Scaled& scaled) {
    const float magic = f.magic(1.0f + float(set) * 0x1p-7f);
    const uint32_t mantissa = ((__float_as_uint(f.s) & 0x007FFFFFu) | 0x00800000u) << (magic < 8192.0f ? 1 : 0);
    uint32_t above = 0xffffffffu, below = 0u;                                // two keys each: twelve bits, then the candidate's number
#pragma unroll
    for (int i = 0; i < kFactorSet; i += 4) {
        const uint32_t p = __byte_perm(mantissa * scaled(i), mantissa * scaled(i + 1), 0x7632) & 0xFFF0FFF0u | uint32_t(i + 0x10000 * (i + 1));
        const uint32_t q = __byte_perm(mantissa * scaled(i + 2), mantissa * scaled(i + 3), 0x7632) & 0xFFF0FFF0u | uint32_t(i + 2 + 0x10000 * (i + 3));
        above = __vimin3_u16x2(above, p, q);
        below = __vimax3_u16x2(below, p, q);
    }
    const uint32_t nearest_above = min(above & 0xFFFFu, above >> 16), nearest_below = max(below & 0xFFFFu, below >> 16);
    const unsigned i = unsigned(set) + ((nearest_above + nearest_below <= 0xFFFFu ? nearest_above : nearest_below) & 15u), widest = max(f.z, 15u - f.z);
    const float a1 = factor_a1(i), a2 = f.a2(inverses[i], magic);
    const int remainder = f.remainder(a1, a2);
    const uint32_t a1_bits = 0x3C003C00u + i * 0x00080008u;
    const __half a2_scaled = __float2half_rn(a2 * f.scale);
    const __half2 a2_pair = __half2half2(a2_scaled), a1_pair = *reinterpret_cast<const __half2*>(&a1_bits);
    const bool exact = (i & 1u) == 0 || widest * (128u + i) < 2048u;
    const uint2 mask = masks[f.z];
    uint32_t differ = 0;
#pragma unroll
    for (int c = 1; c < 16; c += 4) {
        const __half2 want = __floats2half2_rn(__fmul_rn(f.s, float(c)), __fmul_rn(f.s, float(c + 2)));
        const __half2 got = __hmul2(__hmul2(__floats2half2_rn(float(c), float(c + 2)), a1_pair), a2_pair);
        const uint32_t unequal = *reinterpret_cast<const uint32_t*>(&got) ^ *reinterpret_cast<const uint32_t*>(&want);
        differ |= c < 8 ? unequal : unequal & (c == 9 ? mask.x : mask.y);
    }
    return differ == 0 && exact && unsigned(remainder + 512) < 1024u ? factored_field(i, __half_as_ushort(a2_scaled) + (14u << 10), remainder) : 0u;
}

// The field of a step that all lanes of a warp share: the eight nearest of the 128 candidates are checked, two at a time; 0 if none
// gives the weights.
__device__ __forceinline__ uint32_t factor_ranked(const FactorStep& f, const float* inverses, int lane) {
    unsigned key[4];                                                         // |distance| with the candidate's number in the low bits
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const unsigned i = lane + 32 * q;
        const float a1 = factor_a1(i);
        key[q] = (__float_as_uint(__fmaf_rn(-a1, f.a2(inverses[i], f.magic(a1)), f.m)) & 0x7FFFFF80u) | i;
    }
#pragma unroll 1
    for (int round = 0; round < 4; ++round) {
        unsigned nearest[2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            nearest[n] = __reduce_min_sync(0xffffffffu, min(min(key[0], key[1]), min(key[2], key[3])));
#pragma unroll
            for (int q = 0; q < 4; ++q) if (key[q] == nearest[n]) key[q] = 0xffffffffu;
        }
        // lanes 0 to 15 take the sixteen codes of the nearer candidate, lanes 16 to 31 those of the other, with the operations
        // of the factored chain
        const unsigned i = (lane < 16 ? nearest[0] : nearest[1]) & 127u, code = lane & 15;
        const float a1 = factor_a1(i), a2 = f.a2(inverses[i], f.magic(a1));
        const int remainder = f.remainder(a1, a2);
        const uint32_t field = factored_field(i, __half_as_ushort(__float2half_rn(a2 * f.scale * 0x1p14f)), remainder);
        const __half even = __ushort_as_half(uint16_t(0x6400u | i << 3));                                 // a1 * 2^10
        const __half b = __hmul(even, __ushort_as_half(uint16_t(0x8000u | f.z)));                          // -z * a1 * 2^-14
        const __half got = __hmul(__hfma(__ushort_as_half(uint16_t(code)), even, b), __ushort_as_half(uint16_t((field >> 16 & 0x3FFFu) | 0x4000u)));
        const __half want = __float2half_rn(__fmul_rn(float(code) - float(f.z), f.s));
        const unsigned votes = __ballot_sync(0xffffffffu, __half_as_ushort(got) == __half_as_ushort(want) && unsigned(remainder + 512) < 1024u);
        if ((votes & 0xFFFFu) == 0xFFFFu) return __shfl_sync(0xffffffffu, field, 0);
        if (votes >> 16 == 0xFFFFu) return __shfl_sync(0xffffffffu, field, 16);
    }
    return 0u;
}

// The step fields of `per_warp` consecutive blocks per warp.  The nearest of sixteen a1 reproduces all weights in four of five cases
// (weights N(0, 0.02^2)).  Steps that are left go to a list of the CTA, whose warps try the next sixteen candidates, and so on; what is
// left of all 128 (6 in 10^4) gets a whole warp, which ranks them by their distance.  A step that a1 = 1 gives without
// a remainder is found in the first set: its distance is zero, and it passes every check.
//
// What a field promises is that the sequence of operations of the factored chain gives the weights; factor_ranked() runs that very
// sequence.  factor_nearest() does with less: where |d| * a1 has at most eleven significant bits for every d = code - zero the
// chain's first operation is exact, its second rounds d * a1 * a2, and doubling or negating d doubles or negates both that
// and the weight (steps from 2^-12 on keep all of them normal).  So the odd d up to the largest |d| decide, eight instead of
// sixteen; candidates with longer products are left to the other check.
//
// A block in which more than a quarter of the steps lie outside the factored range stays plain: its warps would take the general
// chain all the same.  Every field is written in one store.
//
// Bound by instruction issue (about 370 per 32 steps), on small layers by the chain of sets.  Behind the quantizer 4096 x 12288 16 us,
// 28672 x 12288 70; in a first form (one list of a CTA of sixteen warps, all sixteen codes in every check, a2 only on the coarser of
// the two spacings) 25 and 148, which also left 15 / 64 / 460 plain groups in 10^4 of FP16 / FP32 / positive FP16 weights instead
// of 0.2 / 17 / 119.
__global__ void __launch_bounds__(kFactorThreads, 10)
factor_steps_kernel(uint8_t* native, int64_t blocks, int per_warp, unsigned* flags) {
    constexpr int kFields = 64 * kFactorMaxBlocks * kFactorWarps;
    __shared__ float steps[kFields];                                         // the steps that are left ...
    __shared__ uint16_t where[kFields];                                      // ... and (block of the CTA * 64 + field) * 16 + zero point
    __shared__ float inverses[128];                                          // (constant memory answers one address at a time)
    __shared__ uint2 masks[16];                                              // by zero point: the pairs (9, 11) and (13, 15) that some code has
    __shared__ int counts[kFactorShared];                                    // length of the list behind a set
    __shared__ int any;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < 128) inverses[tid] = kFactorTable.inverse[tid];
    if (tid < kFactorShared) counts[tid] = 0;
    if (tid == kFactorShared) any = 0;
    if (tid >= 32 && tid < 48) {
        const int z = tid - 32, widest = max(z, 15 - z);
        masks[z] = make_uint2((widest >= 9 ? 0xFFFFu : 0u) | (widest >= 11 ? 0xFFFF0000u : 0u), (widest >= 13 ? 0xFFFFu : 0u) | (widest >= 15 ? 0xFFFF0000u : 0u));
    }
    __syncthreads();
    const int64_t cta0 = int64_t(blockIdx.x) * kFactorWarps * per_warp;
    auto fields = [&](int block) { return reinterpret_cast<uint32_t*>(native + (cta0 + block) * kBlockBytes + kStepOffset); };
    bool found = false;
    auto append = [&](int list, bool yes, float s, uint32_t w) {             // (called by whole warps)
        const unsigned votes = __ballot_sync(0xffffffffu, yes);
        int base = 0;
        if (lane == 0 && votes) base = atomicAdd(&counts[list], __popc(votes));
        base = __shfl_sync(0xffffffffu, base, 0) + __popc(votes & ((1u << lane) - 1u));
        if (yes) {
            steps[base] = s;
            where[base] = uint16_t(w);
        }
    };
    const int mine = int(min(int64_t(kFactorWarps) * per_warp, blocks - cta0));
    uint32_t next[2], next_zero[2];
    auto fetch = [&](int b) {
        const uint32_t* const at = fields(b);
        const uint8_t* const zeros = reinterpret_cast<const uint8_t*>(at) + (kZeroOffset - kStepOffset);
        next[0] = at[lane]; next[1] = at[lane + 32];
        next_zero[0] = zeros[lane >> 1]; next_zero[1] = zeros[16 + (lane >> 1)];
    };
    if (warp < mine) fetch(warp);
#pragma unroll 1
    for (int b = warp; b < mine; b += kFactorWarps) {
        uint32_t* const at = fields(b);
        const uint32_t have[2] = {next[0], next[1]}, zero[2] = {next_zero[0], next_zero[1]};
        if (b + kFactorWarps < mine) fetch(b + kFactorWarps);
        bool wanted[2];
        int misses = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float s = __uint_as_float(have[h]);                        // (factored fields are negative)
            wanted[h] = s >= 0x1p-12f && s < 3.99f;
            misses += __popc(__ballot_sync(0xffffffffu, int32_t(have[h]) >= 0 && !wanted[h]));
        }
        if (misses > kFactorMisses) continue;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const uint32_t z = ((h ? zero[1] : zero[0]) >> (4 * (lane & 1))) & 15u;
            const bool want = h ? wanted[1] : wanted[0];
            const float s = want ? __uint_as_float(h ? have[1] : have[0]) : 1.0f;
            const uint32_t field = factor_nearest(FactorStep(s, z), 0, inverses, masks, [](int i) { return kFactorTable.scaled[i]; });
            if (want && field) {
                at[lane + 32 * h] = field;
                found = true;
            }
            append(0, want && !field, s, uint32_t(b * 64 + 32 * h + lane) * 16 + z);
        }
    }
    // The list is closed up in place: the entries of a round of the CTA have been read before its first one is written, and at most
    // as many are written as have been read.
#pragma unroll 1
    for (int n = 1; n < kFactorShared; ++n) {
        __syncthreads();
        const int count = counts[n - 1];
        if (count == 0) break;
#pragma unroll 1
        for (int first = 0; first < count; first += kFactorThreads) {
            const bool active = first + tid < count;
            const float s = steps[active ? first + tid : first];
            const uint32_t w = where[active ? first + tid : first];
            __syncthreads();
            if (first + 32 * warp < count) {
                const int set = n * kFactorSet;
                const uint32_t field = factor_nearest(FactorStep(s, w & 15u), set, inverses, masks, [set](int i) { return kFactorTable.scaled[set + i]; });
                if (active && field) {
                    fields(int(w >> 10))[w >> 4 & 63] = field;
                    found = true;
                }
                append(n, active && !field, s, w);
            }
        }
    }
    __syncthreads();
    for (int first = 32 * warp; first < counts[kFactorShared - 1]; first += kFactorThreads) {
        bool open = first + lane < counts[kFactorShared - 1];
        const float s = steps[open ? first + lane : first];
        const uint32_t w = where[open ? first + lane : first];
#pragma unroll 1
        for (int set = kFactorShared * kFactorSet; set < 128 && __any_sync(0xffffffffu, open); set += kFactorSet) {
            const uint32_t field = factor_nearest(FactorStep(s, w & 15u), set, inverses, masks, [set](int i) { return kFactorTable.scaled[set + i]; });
            if (open && field) {
                fields(int(w >> 10))[w >> 4 & 63] = field;
                found = true;
                open = false;
            }
        }
        for (unsigned left = __ballot_sync(0xffffffffu, open); left; left &= left - 1) {
            const int from = __ffs(left) - 1;
            const uint32_t entry = __shfl_sync(0xffffffffu, w, from);
            const uint32_t field = factor_ranked(FactorStep(__shfl_sync(0xffffffffu, s, from), entry & 15u), inverses, lane);
            if (lane == 0 && field) {
                fields(int(entry >> 10))[entry >> 4 & 63] = field;
                found = true;
            }
        }
    }
    if (flags) {
        if (__any_sync(0xffffffffu, found) && lane == 0) any = 1;
        __syncthreads();
        if (tid == 0 && any && !(*static_cast<volatile unsigned*>(flags) & kQuantFactored)) atomicOr(flags, kQuantFactored);
    }
}

}  // namespace b2
