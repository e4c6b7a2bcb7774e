// Conversion kernels between floating-point weights, the checkpoint tensors and the native image.
//
// quantize_kernel reads every weight once (2 or 4 bytes) and writes everything a layer keeps of it - packed codes, FP32
// step, zero point, native image - in the same pass.  The same steps as separate
// elementwise and reduction passes over an FP32 copy move about forty bytes per weight.  Measured on 4096 x 12288
// FP16: 1690 us for the whole conversion as separate passes (with packing, value checks and relayout), 43 us here
// (2.3 TB/s of input, 3.7 TB/s with everything written): bound by the instructions of range and rounding and, between them, by
// the wait for the weights (nine CTAs of four warps on an SM instead of eight: 44.8 -> 43.2; FP32 weights ten, 46.8 -> 45.2).
#pragma once
#include <cfloat>
#include <type_traits>
#include "layout.cuh"

namespace b2 {

struct QuantizeArgs {
    const void* weight;      // [N, K] contiguous
    uint8_t* codes;          // [N, K], may be null
    int32_t* packed;         // [N, ceil(K/8)], may be null
    float* scales;           // [N, ceil(K/64)]
    int32_t* zeros;          // [N, ceil(K/64)]
    uint8_t* native;         // native image, may be null
    unsigned* flags;         // OR of kQuant*; zero before the launch
    Dims d;
};

// Eight consecutive weights of a row, held as they are stored; columns >= valid are zero (they take part in the
// range, as the zero padding of the reference's last group does).
template <typename T> struct Eight;
template <> struct Eight<float> {
    float v[8];
    template <bool VEC> __device__ __forceinline__ void load(const float* src, int valid) {
        if (VEC && valid > 0) {            // K % 8 == 0: a word is whole or absent
            const float4 a = __ldcs(reinterpret_cast<const float4*>(src)), b = __ldcs(reinterpret_cast<const float4*>(src) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = c < valid ? __ldg(src + c) : 0.0f;
        }
    }
    __device__ __forceinline__ void range(float& lo, float& hi, bool& finite) const {
        float poison = 0.0f;                                 // NaN as soon as one weight is not finite
        lo = hi = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            lo = fminf(lo, v[c]);
            hi = fmaxf(hi, v[c]);
            poison = fmaf(v[c], 0.0f, poison);
        }
        finite = finite && poison == 0.0f;
    }
    __device__ __forceinline__ void widen(float (&f)[8]) const {
#pragma unroll
        for (int c = 0; c < 8; ++c) f[c] = v[c];
    }
};
template <> struct Eight<__half> {
    uint32_t p[4];
    template <bool VEC> __device__ __forceinline__ void load(const __half* src, int valid) {
        if (VEC && valid > 0) {
            const uint4 a = __ldcs(reinterpret_cast<const uint4*>(src));
            p[0] = a.x; p[1] = a.y; p[2] = a.z; p[3] = a.w;
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t lo = 2 * c < valid ? __half_as_ushort(__ldg(src + 2 * c)) : 0u;
                const uint32_t hi = 2 * c + 1 < valid ? __half_as_ushort(__ldg(src + 2 * c + 1)) : 0u;
                p[c] = lo | hi << 16;
            }
        }
    }
    __device__ __forceinline__ __half2 pair(int c) const { return *reinterpret_cast<const __half2*>(&p[c]); }
    __device__ __forceinline__ void range(float& lo, float& hi, bool& finite) const {      // two weights per instruction
        const __half2 zero = __half2half2(__ushort_as_half(0));
        __half2 l = zero, h = zero;                          // (a NaN stays in both, an infinity in one)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            l = __hmin2_nan(l, pair(c));
            h = __hmax2_nan(h, pair(c));
        }
        const float2 lf = __half22float2(l), hf = __half22float2(h);
        lo = fminf(lf.x, lf.y);
        hi = fmaxf(hf.x, hf.y);
        finite = finite && (hf.x - lf.x) + (hf.y - lf.y) < 1e6f;
    }
    __device__ __forceinline__ void widen(float (&f)[8]) const {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float2 w = __half22float2(pair(c));
            f[2 * c] = w.x; f[2 * c + 1] = w.y;
        }
    }
};

__device__ __forceinline__ float reciprocal(float v) {       // to one unit in the last place
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// Packed codes of eight weights: code = clamp(round_half_even(fl(fl(w / step) + zero)), 0, 15).
//
// The sum is first taken as w * (1 / step) + zero with the approximate reciprocal: |w / step| is at most 15 plus
// rounding, so it is off by less than 2^-17 together with the two roundings of the definition.  Only a sum that close
// to a half-integer can round to another code; where one of the eight is (one word in ~10^4), or where the
// reciprocal of the step is not a normal number, the eight weights are divided.  Only there, too, can a code be outside 0..15:
// the ends of the range are at -0.5 and 15.5.
//
// Rounding is an addition of 1.5 * 2^23, whose ulp is 1, in the fma that forms the sum: half-to-even for sums this small, and
// the code is then in the low byte (rintf and the float-to-int conversion run at an eighth of the rate of an addition).
constexpr float kRoundMagic = 12582912.0f;
__device__ __forceinline__ int code_of(float u) { return __float_as_int(u) - 0x4B400000; }
// The eight codes of a word in the low halves of bytes: columns 0, 2, 4, 6 and columns 1, 3, 5, 7.
struct Codes {
    uint32_t even, odd;
    __device__ __forceinline__ uint32_t reference() const { return even + (odd << 4); }            // nibble c = column c
    __device__ __forceinline__ uint32_t native() const { return __byte_perm(even | even >> 4, odd | odd >> 4, 0x6420); }
};
__device__ __forceinline__ uint32_t low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
__device__ __forceinline__ Codes quantize_word(const float (&v)[8], float step, float zero) {
    const float inverse = reciprocal(step), base = zero + kRoundMagic;
    float off = step < 0x1p100f ? 0.0f : 1.0f;              // largest distance of a sum from the integer it rounds to
    uint32_t q[8];
#pragma unroll
    for (int c = 0; c < 8; c += 2) {                        // two weights per instruction, each rounded as if alone
        float u0, u1, d0, d1;
        asm("{\n\t.reg .b64 u, r, v, i, z;\n\t"
            "mov.b64 v, {%4, %5};\n\tmov.b64 i, {%6, %6};\n\tmov.b64 z, {%7, %7};\n\t"
            "fma.rn.f32x2 u, v, i, z;\n\tsub.rn.f32x2 r, z, u;\n\tfma.rn.f32x2 r, v, i, r;\n\t"
            "mov.b64 {%0, %1}, u;\n\tmov.b64 {%2, %3}, r;\n\t}"
            : "=f"(u0), "=f"(u1), "=f"(d0), "=f"(d1)
            : "f"(v[c]), "f"(v[c + 1]), "f"(inverse), "f"(base));
        asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(off) : "f"(off), "f"(d0), "f"(d1));
        q[c] = __float_as_uint(u0);
        q[c + 1] = __float_as_uint(u1);
    }
    if (off > 0.5f - 0x1p-16f) {
#pragma unroll
        for (int c = 0; c < 8; ++c) q[c] = uint32_t(min(max(code_of(__fadd_rn(__fadd_rn(__fdiv_rn(v[c], step), zero), kRoundMagic)), 0), 15));
    }
    return Codes{low_bytes(q[0], q[2], q[4], q[6]), low_bytes(q[1], q[3], q[5], q[7])};
}

// v / 15, correctly rounded, in two operations: v times the high part of 1/15 plus (v times the low part), a division by a constant
// after Brisebarre, Muller and Raina (IEEE Trans. Computers 53, 2004).  Equal to the division for all 2^23 mantissas as long as the
// small product is a normal number; smaller and larger values are divided.
__device__ __forceinline__ float fifteenth(float v) {
    const float q = __fmaf_rn(v, 0x1.111112p-4f, __fmul_rn(v, -0x1.dddddep-29f));
    return fabsf(v) > 0x1p-90f && fabsf(v) < 0x1p120f ? q : __fdiv_rn(v, 15.0f);
}

// clamp(round_half_even(fl(-lo / step)), 0, 15): as for a code, the quotient by the approximate reciprocal decides unless it is
// close to a half-integer.
__device__ __forceinline__ float zero_point(float lo, float step) {
    const float inverse = reciprocal(step), u = __fmaf_rn(-lo, inverse, kRoundMagic), r = __fsub_rn(u, kRoundMagic);
    const float off = fabsf(__fmaf_rn(-lo, inverse, -r));
    const float zero = step < 0x1p100f && off < 0.5f - 0x1p-16f ? r : rintf(__fdiv_rn(-lo, step));
    return fminf(fmaxf(zero, 0.0f), 15.0f);
}

// One CTA of four warps per 16 x 256 block; warp w takes the rows w, w + 4, w + 8 and w + 12, lane 8t + i word i of
// group t.  The eight lanes of a group reduce the ranges of the four rows together: each exchange halves the number
// of rows a lane carries, so that lane i ends with the range of row i % 4 and computes that row's step and zero
// point (IEEE divisions are what this kernel could least afford to repeat in every lane), which the others fetch.
template <typename T, bool VEC>
__global__ void __launch_bounds__(128, sizeof(T) == 2 ? 9 : 10)
quantize_kernel(const QuantizeArgs a) {
    constexpr unsigned kAll = 0xffffffffu;
    const Dims& d = a.d;
    const int nt = int(blockIdx.x) / d.kb, kb = int(blockIdx.x) - nt * d.kb;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane >> 3, wi = lane & 7;
    const int k0 = kb * kBlockCols + lane * 8, grp = kb * 4 + t;
    const int valid = min(8, d.k - k0);
    Eight<T> v[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int row = nt * 16 + w + 4 * p;
        v[p].template load<VEC>(static_cast<const T*>(a.weight) + int64_t(row) * d.k + k0, row < d.n ? valid : 0);
    }
    float lo[4], hi[4];
    bool finite = true;
#pragma unroll
    for (int p = 0; p < 4; ++p) v[p].range(lo[p], hi[p], finite);
    unsigned found = finite ? 0u : kQuantNonFinite;
    const bool b0 = wi & 1, b1 = wi & 2;
    auto exchange = [&](float& keep, float mine, float give, int mask, bool low) {
        const float got = __shfl_xor_sync(kAll, give, mask);
        keep = low ? fminf(mine, got) : fmaxf(mine, got);
    };
#pragma unroll
    for (int p = 0; p < 4; p += 2) {                         // rows p and p + 1 -> row p + b0
        exchange(lo[p], b0 ? lo[p + 1] : lo[p], b0 ? lo[p] : lo[p + 1], 1, true);
        exchange(hi[p], b0 ? hi[p + 1] : hi[p], b0 ? hi[p] : hi[p + 1], 1, false);
    }
    exchange(lo[0], b1 ? lo[2] : lo[0], b1 ? lo[0] : lo[2], 2, true);
    exchange(hi[0], b1 ? hi[2] : hi[0], b1 ? hi[0] : hi[2], 2, false);
    exchange(lo[0], lo[0], lo[0], 4, true);                  // lanes i and i + 4 hold the same row
    exchange(hi[0], hi[0], hi[0], 4, false);
    // two quotients and a difference, each rounded; never below the smallest normal FP32; 1 for an all-zero group
    float my_step = fmaxf(__fsub_rn(fifteenth(hi[0]), fifteenth(lo[0])), FLT_MIN);
    if (hi[0] == 0.0f && lo[0] == 0.0f) my_step = 1.0f;
    const float my_zero = zero_point(lo[0], my_step);
    uint8_t* block = a.native ? a.native + (int64_t(kb) * d.n16 + nt) * kBlockBytes : nullptr;
    {   // lane i < 4 of a group keeps the books of row w + 4i
        const int r = w + 4 * (wi & 3), row = nt * 16 + r;
        const bool real = row < d.n && grp < d.groups;
        if (wi < 4) {
            if (real) {
                if (__half2float(__float2half_rn(my_step)) != my_step) found |= kQuantStepNotFp16;
                a.scales[int64_t(row) * d.groups + grp] = my_step;
                a.zeros[int64_t(row) * d.groups + grp] = int32_t(my_zero);
            }
            if (block) reinterpret_cast<uint32_t*>(block + kStepOffset)[(4 * (r & 7) + t) * 2 + (r >> 3)] = real ? __float_as_uint(my_step) : kPaddingField;
        }
        // zero points of rows r and r + 8 share a byte
        const unsigned z = real ? unsigned(int(my_zero)) : 0u, z8 = __shfl_xor_sync(kAll, z, 2);
        if (block && wi < 2) block[kZeroOffset + 4 * (r & 7) + t] = uint8_t(z | z8 << 4);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int r = w + 4 * p, row = nt * 16 + r;
        const float step = __shfl_sync(kAll, my_step, (lane & 24) | p), zero = __shfl_sync(kAll, my_zero, (lane & 24) | p);
        const bool real = row < d.n && grp < d.groups;
        float f[8];
        v[p].widen(f);
        const Codes codes = quantize_word(f, step, zero);
        uint32_t ref = codes.reference();
        if (!VEC && valid < 8) ref &= valid > 0 ? 0xffffffffu >> (32 - 4 * valid) : 0u;
        if (real && valid > 0) {
            if (a.packed) a.packed[int64_t(row) * d.words + (k0 >> 3)] = int32_t(ref);
            if (a.codes) {
                uint8_t* dst = a.codes + int64_t(row) * d.k + k0;
                if constexpr (VEC) {
                    const uint32_t even = ref & 0x0F0F0F0Fu, odd = (ref >> 4) & 0x0F0F0F0Fu;
                    *reinterpret_cast<uint2*>(dst) = make_uint2(__byte_perm(even, odd, 0x5140), __byte_perm(even, odd, 0x7362));
                } else {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        if (c < valid) dst[c] = uint8_t((ref >> (4 * c)) & 15u);
                }
            }
        }
        if (block) {                   // rows and groups that do not exist: code 0; columns beyond K: the zero point
            const uint32_t fill = uint32_t(int(zero));
            const uint32_t nat = !real ? 0u : valid >= 8 ? codes.native() : permute_word(ref, max(valid, 0), fill);
            reinterpret_cast<uint32_t*>(block)[(2 * (r >> 3) + (wi >> 2)) * 128 + (4 * (r & 7) + t) * 4 + (wi & 3)] = nat;
        }
    }
    // nearly every warp of a layer finds a step that FP16 cannot hold: only the first ones write the word
    found = __reduce_or_sync(kAll, found);
    if (lane == 0 && (found & ~*static_cast<volatile unsigned*>(a.flags))) atomicOr(a.flags, found);
}

__device__ __forceinline__ float dequantize_one(uint32_t code, int zero, float step) {
    return __fmul_rn(float(int(code) - zero), step);
}

template <typename Out, int V>
__device__ __forceinline__ void store_unit(Out* dst, const float (&v)[V]) {
    if constexpr (V == 1) {
        if constexpr (sizeof(Out) == 2) *dst = __float2half_rn(v[0]);
        else *dst = v[0];
    } else if constexpr (sizeof(Out) == 2) {           // V = 8
        uint32_t p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            p[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        __stcs(reinterpret_cast<uint4*>(dst), make_uint4(p[0], p[1], p[2], p[3]));
    } else {                                            // V = 4
        __stcs(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
    }
}

// Checkpoint tensors -> FP32.  A warp takes kStateRuns runs of 256 columns of a row (consecutive runs, so nearly always one row): lane i
// loads word i of a run, lanes 0..3 its four steps and zero points, and the lanes of a store, four columns each (VEC; else one), fetch
// theirs by shuffle: a word is loaded once, a store is 512 (128) consecutive bytes, and a run costs no division.  Bound by the stores:
// 6144 x 4096 17.4 us (6.6 TB/s into L2 and memory; a fill of the output 15.0), 4096 x 12288 34.8 (28.7); with a thread per four
// columns that found its row, word, step and zero point by itself, bound by instructions, 24.0 and 46.5.  Codes become floats as
// 2^23 + code, from which 2^23 + zero is subtracted exactly.
constexpr int kStateRuns = 4;
constexpr int kStateWarps = 8;
template <bool VEC>
__global__ void __launch_bounds__(kStateWarps * 32)
dequantize_state_kernel(const int32_t* __restrict__ packed, const float* __restrict__ scales, const int32_t* __restrict__ zeros, Dims d,
                        float* __restrict__ out, int64_t ldo) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned first = (blockIdx.x * kStateWarps + (threadIdx.x >> 5)) * kStateRuns, total = unsigned(d.n) * unsigned(d.kb);
    if (first >= total) return;
    int row = int(first / unsigned(d.kb)), run = int(first - unsigned(row) * unsigned(d.kb));
    const int64_t row0 = row;
    const int run0 = run;
    uint32_t word[kStateRuns];
    float step[kStateRuns];
    int zero[kStateRuns];
#pragma unroll
    for (int i = 0; i < kStateRuns; ++i) {
        word[i] = 0; step[i] = 0.0f; zero[i] = 0;
        if (row < d.n) {
            const int w = run * 32 + lane, g = run * 4 + lane;
            if (w < d.words) word[i] = uint32_t(__ldg(packed + int64_t(row) * d.words + w));
            if (lane < 4 && g < d.groups) {
                step[i] = __ldg(scales + int64_t(row) * d.groups + g);
                zero[i] = __ldg(zeros + int64_t(row) * d.groups + g) & 15;         // as the image holds it
            }
        }
        if (++run == d.kb) { run = 0; ++row; }
    }
    row = int(row0);
    run = run0;
#pragma unroll
    for (int i = 0; i < kStateRuns; ++i) {
        if (row >= d.n) break;
        constexpr int V = VEC ? 4 : 1, kStores = 8 / V;
        float* dst = out + int64_t(row) * ldo + run * kBlockCols + lane * V;
#pragma unroll
        for (int j = 0; j < kStores; ++j) {
            const int col = j * 32 * V + lane * V, grp = VEC ? col >> 6 : j >> 1;         // of the run
            const uint32_t codes = __shfl_sync(kAll, word[i], col >> 3) >> (4 * (col & 7));
            const float s = __shfl_sync(kAll, step[i], grp), base = __int_as_float(0x4B000000 + __shfl_sync(kAll, zero[i], grp));
            float v[V];
#pragma unroll
            for (int c = 0; c < V; ++c)
                v[c] = __fmul_rn(__fsub_rn(__uint_as_float(0x4B000000u | ((codes >> (4 * c)) & 15u)), base), s);
            if (run * kBlockCols + col < d.k) {
                if constexpr (VEC) __stcs(reinterpret_cast<float4*>(dst + j * 128), make_float4(v[0], v[1], v[2], v[3]));
                else __stcs(dst + j * 32, v[0]);
            }
        }
        if (++run == d.kb) { run = 0; ++row; }
    }
}

// Unit = V consecutive columns of a row, one 16-byte store (V = 1: one element, for rows that are not whole
// units); the lanes of a warp write consecutive units.  A thread takes kDequantUnits units a CTA apart so that their loads are in
// flight together.
constexpr int kDequantUnits = 4;
template <typename Out, int V>
__global__ void __launch_bounds__(256)
dequantize_kernel(const uint8_t* __restrict__ native, Dims d, Out* __restrict__ out, int64_t ldo) {
    const unsigned per_row = unsigned(d.k) / V;
    const int64_t total = int64_t(d.n) * per_row;
    const int64_t u0 = int64_t(blockIdx.x) * (256 * kDequantUnits) + threadIdx.x;
    uint32_t word[kDequantUnits];
    float step[kDequantUnits];
    int zero[kDequantUnits];
#pragma unroll
    for (int i = 0; i < kDequantUnits; ++i) {
        const int64_t u = u0 + i * 256;
        word[i] = 0; step[i] = 0.0f; zero[i] = 0;
        if (u < total) {
            const int row = int(unsigned(u) / per_row), col = int(unsigned(u) - unsigned(row) * per_row) * V;
            const WordRef w = locate(d, row, col >> 3);
            const uint8_t* base = native + w.block;
            word[i] = __ldg(reinterpret_cast<const uint32_t*>(base) + w.word);
            step[i] = field_step(__ldg(reinterpret_cast<const uint32_t*>(base + kStepOffset) + w.meta));
            zero[i] = (__ldg(base + kZeroOffset + (w.meta >> 1)) >> (4 * (w.meta & 1))) & 15;
        }
    }
#pragma unroll
    for (int i = 0; i < kDequantUnits; ++i) {
        const int64_t u = u0 + i * 256;
        if (u >= total) break;
        const int row = int(unsigned(u) / per_row), col = int(unsigned(u) - unsigned(row) * per_row) * V;
        float v[V];
#pragma unroll
        for (int c = 0; c < V; ++c) {
            const int cc = (col & 7) + c;
            v[c] = dequantize_one((word[i] >> (4 * nibble_slot(cc))) & 15u, zero[i], step[i]);
        }
        store_unit<Out, V>(out + int64_t(row) * ldo + col, v);
    }
}

}  // namespace b2
