// C ABI of the load-time conversions: quantizer, packer, relayout to and from the native image, dequantizers.
// Declarations and the per-function reference citations are in include/b2_w4a16.h.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/b2_w4a16.h"
#include "factor_steps.cuh"
#include "host_common.cuh"
#include "layout.cuh"
#include "layout_kernels.cuh"
#include "quantize_kernels.cuh"

namespace {

using b2host::after_launch;
using b2host::check_dims;
using b2host::fail;

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

template <typename Out>
int run_dequantize(const uint8_t* native, const b2::Dims& d, Out* out, int64_t ldo, cudaStream_t s) {
    constexpr int kVec = 16 / int(sizeof(Out));
    constexpr int64_t kPerCta = 256 * b2::kDequantUnits;
    const int64_t elements = int64_t(d.n) * d.k;
    // 16-byte stores need rows that are whole, aligned units
    if (d.k % kVec == 0 && ldo % kVec == 0 && aligned16(out)) {
        const int64_t units = elements / kVec;
        b2::dequantize_kernel<Out, kVec><<<unsigned((units + kPerCta - 1) / kPerCta), 256, 0, s>>>(native, d, out, ldo);
    } else {
        b2::dequantize_kernel<Out, 1><<<unsigned((elements + kPerCta - 1) / kPerCta), 256, 0, s>>>(native, d, out, ldo);
    }
    return after_launch("dequantize_kernel");
}

int run_dequantize_state(const int32_t* packed, const float* scales, const int32_t* zeros, const b2::Dims& d, float* out, int64_t ldo,
                         cudaStream_t s) {
    constexpr int64_t kRuns = int64_t(b2::kStateWarps) * b2::kStateRuns;
    const unsigned ctas = unsigned((int64_t(d.n) * d.kb + kRuns - 1) / kRuns);
    if (d.k % 4 == 0 && ldo % 4 == 0 && aligned16(out))
        b2::dequantize_state_kernel<true><<<ctas, b2::kStateWarps * 32, 0, s>>>(packed, scales, zeros, d, out, ldo);
    else
        b2::dequantize_state_kernel<false><<<ctas, b2::kStateWarps * 32, 0, s>>>(packed, scales, zeros, d, out, ldo);
    return after_launch("dequantize_state_kernel");
}

// Blocks of a warp: as few as let all warps run at once (40 on an SM; a 4096 x 12288 layer has three), for the shortest chain of
// sets, up to eight, with which the lists of later sets fill most of a warp.
int run_factor_steps(uint8_t* native, const b2::Dims& d, unsigned* flags, cudaStream_t s) {
    constexpr int64_t kResident = 148 * 40;
    const int64_t blocks = int64_t(d.n16) * d.kb;
    const int64_t per_warp = std::min<int64_t>(b2::kFactorMaxBlocks, (blocks + kResident - 1) / kResident);
    const int64_t per_cta = per_warp * b2::kFactorWarps;
    b2::factor_steps_kernel<<<unsigned((blocks + per_cta - 1) / per_cta), b2::kFactorThreads, 0, s>>>(native, blocks, int(per_warp), flags);
    return after_launch("factor_steps_kernel");
}

template <typename T>
int run_quantize(const b2::QuantizeArgs& a, cudaStream_t s) {
    const unsigned blocks = unsigned(int64_t(a.d.n16) * a.d.kb);
    const bool vec = a.d.k % 8 == 0 && aligned16(a.weight) && reinterpret_cast<uintptr_t>(a.codes) % 8 == 0;
    if (vec) b2::quantize_kernel<T, true><<<blocks, 128, 0, s>>>(a);
    else b2::quantize_kernel<T, false><<<blocks, 128, 0, s>>>(a);
    if (int rc = after_launch("quantize_kernel")) return rc;
    return a.native ? run_factor_steps(a.native, a.d, a.flags, s) : B2_OK;
}

}  // namespace

extern "C" {

int64_t b2_w4a16_native_bytes(int64_t n, int64_t k) {
    if (check_dims(n, k) != B2_OK) return 0;
    return b2::native_bytes(b2::make_dims(n, k));
}

int b2_w4a16_repack(const int32_t* packed, const float* scales, const int32_t* zeros, int64_t n,
                    int64_t k, void* native, void* stream) {
    if (!packed || !scales || !zeros || !native) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    if (reinterpret_cast<uintptr_t>(native) % 256) return fail(B2_ERR_ARGUMENT, "native image must be 256-byte aligned");
    const b2::Dims d = b2::make_dims(n, k);
    const int64_t blocks = int64_t(d.n16) * d.kb;
    b2::repack_kernel<<<unsigned(blocks), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        packed, scales, zeros, d, static_cast<uint8_t*>(native));
    if (int rc = after_launch("repack_kernel")) return rc;
    return b2_w4a16_factor_steps(native, n, k, stream);
}

int b2_w4a16_factor_steps(void* native, int64_t n, int64_t k, void* stream) {
    if (!native) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    if (reinterpret_cast<uintptr_t>(native) % 4) return fail(B2_ERR_ARGUMENT, "misaligned native image");
    const b2::Dims d = b2::make_dims(n, k);
    return run_factor_steps(static_cast<uint8_t*>(native), d, nullptr, static_cast<cudaStream_t>(stream));
}

int b2_w4a16_image_flags(const void* native, int64_t n, int64_t k, unsigned* flags, void* stream) {
    if (!native || !flags) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    if (reinterpret_cast<uintptr_t>(native) % 4) return fail(B2_ERR_ARGUMENT, "misaligned native image");
    const b2::Dims d = b2::make_dims(n, k);
    const int64_t fields = int64_t(d.n16) * d.kb * 64;
    b2::image_flags_kernel<<<unsigned((fields + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint8_t*>(native), d, flags);
    return after_launch("image_flags_kernel");
}

int b2_w4a16_unrepack(const void* native, int64_t n, int64_t k, int32_t* packed, float* scales,
                      int32_t* zeros, void* stream) {
    if (!packed || !scales || !zeros || !native) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    const b2::Dims d = b2::make_dims(n, k);
    const int64_t total = int64_t(d.n) * d.words;
    b2::unrepack_kernel<<<unsigned((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t*>(native), d, packed, scales, zeros);
    return after_launch("unrepack_kernel");
}

int b2_w4a16_pack(const uint8_t* codes, int64_t n, int64_t k, int32_t* packed, void* stream) {
    if (!codes || !packed) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    const b2::Dims d = b2::make_dims(n, k);
    const int64_t total = int64_t(d.n) * d.words;
    b2::pack_kernel<<<unsigned((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(codes, d, packed);
    return after_launch("pack_kernel");
}

int b2_w4a16_quantize(const void* weight, int weight_bits, int64_t n, int64_t k, uint8_t* codes, int32_t* packed, float* scales,
                      int32_t* zeros, void* native, unsigned* flags, void* stream) {
    if (!weight || !scales || !zeros || !flags) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (weight_bits != 16 && weight_bits != 32) return fail(B2_ERR_ARGUMENT, "weight_bits must be 16 or 32");
    if (int rc = check_dims(n, k)) return rc;
    if (reinterpret_cast<uintptr_t>(weight) % (weight_bits / 8)) return fail(B2_ERR_ARGUMENT, "misaligned weight");
    if (reinterpret_cast<uintptr_t>(native) % 256) return fail(B2_ERR_ARGUMENT, "native image must be 256-byte aligned");
    b2::QuantizeArgs a;
    a.weight = weight;
    a.codes = codes; a.packed = packed; a.scales = scales; a.zeros = zeros;
    a.native = static_cast<uint8_t*>(native);
    a.flags = flags;
    a.d = b2::make_dims(n, k);
    return weight_bits == 16 ? run_quantize<__half>(a, static_cast<cudaStream_t>(stream)) : run_quantize<float>(a, static_cast<cudaStream_t>(stream));
}

int b2_w4a16_dequantize(const void* native, int64_t n, int64_t k, float* out, int64_t ldo, void* stream) {
    if (!native || !out) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    if (ldo < k) return fail(B2_ERR_ARGUMENT, "ldo must be at least k");
    return run_dequantize<float>(static_cast<const uint8_t*>(native), b2::make_dims(n, k), out, ldo, static_cast<cudaStream_t>(stream));
}

int b2_w4a16_dequantize_fp16(const void* native, int64_t n, int64_t k, void* out, int64_t ldo, void* stream) {
    if (!native || !out) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    if (ldo < k) return fail(B2_ERR_ARGUMENT, "ldo must be at least k");
    return run_dequantize<__half>(static_cast<const uint8_t*>(native), b2::make_dims(n, k), static_cast<__half*>(out), ldo,
                                  static_cast<cudaStream_t>(stream));
}

int b2_w4a16_dequantize_state(const int32_t* packed, const float* scales, const int32_t* zeros, int64_t n, int64_t k, float* out,
                              int64_t ldo, void* stream) {
    if (!packed || !scales || !zeros || !out) return fail(B2_ERR_ARGUMENT, "null pointer");
    if (int rc = check_dims(n, k)) return rc;
    if (ldo < k) return fail(B2_ERR_ARGUMENT, "ldo must be at least k");
    return run_dequantize_state(packed, scales, zeros, b2::make_dims(n, k), out, ldo, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
