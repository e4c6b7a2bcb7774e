// Two row tiles per CTA: the tile kernel (tile_kernel.cuh) for 9 to 16 rows of x where a layer has one to two row tiles for every SM.
//
// Sixteen rows of x of a 4096-column layer take 130 KB of shared memory, so that one CTA of the tile kernel fills an SM and a
// layer of 256 row tiles runs in two waves, each of which fetches x again.  Here a CTA takes two neighbouring tiles, the whole K
// range of both: one wave, x staged once, every fragment of x that a warp reads multiplied with the weights of both tiles, and one
// bulk copy per 256 columns for the two (neighbouring) native blocks.  As in the tile kernel a unit is half a block, the warps take
// consecutive units, the first of which each decodes (of its first tile) before the previous kernel has ended, and the warps' sums are
// added in warp order (the same bits).  The sums' tiles reuse the weights' shared memory.  Bound by the trip of x to every SM (2 us for
// 128 KB) between the previous kernel's end and the products.  us in a chain of launches at M = 9 / 16, one tile / two per CTA, on layers
// that the automatic route leaves to the tile kernel: 4096 x 4096 10.2 / 9.7 -> 7.0 / 7.3, 4096 x 2048 4.5 / 4.9 -> 4.4 / 4.6, 2560 x 2048 4.4 / 4.8 ->
// 4.0 / 4.4.  (Up to 8 rows two CTAs of the tile kernel share an SM and are ahead: 4096 x 4096 at M = 1 / 4 5.1 / 5.4 against 5.4 / 5.5.)
// 128 registers; spills of 12 to 24 bytes (stores).
#pragma once
#include "tile_kernel.cuh"

namespace b2 {

constexpr int kTilePairWarps = 16, kTilePairMinBlocks = 8;            // (the sums of all warps fit over eight blocks)
__host__ __device__ constexpr int tile_pair_smem_bytes(int kb) {
    return ((kb * 8 + 127) / 128) * 128 + kb * (2 * kBlockBytes + 4 * tile_x_chunk_bytes(16));
}

template <int STEPS>
__global__ void __launch_bounds__(kTilePairWarps * 32, 1)
w4a16_tile_pair_kernel(const TileArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int MT = 2, kChunk = tile_x_chunk_bytes(MT * 8), kPair = 2 * kBlockBytes;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int nt = 2 * blockIdx.x, tiles = min(2, a.n16 - nt);
    uint8_t* blocks = smem + ((a.kb * 8 + 127) / 128) * 128;
    uint8_t* xs = blocks + a.kb * kPair;
    static_assert(kTilePairWarps * 2 * MT * 512 <= kTilePairMinBlocks * kPair, "the sums fit over the weights");
    float4* red = reinterpret_cast<float4*>(blocks);            // [warp][tile][MT][32], once the weights have been used
    const uint32_t bar0 = smem_u32(smem);

    if (threadIdx.x == 0) {
        for (int b = 0; b < a.kb; ++b) mbar_init(bar0 + b * 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        const uint8_t* src = a.native + int64_t(nt) * kBlockBytes;
        const int64_t stride = int64_t(a.n16) * kBlockBytes;
        for (int b = 0; b < a.kb; ++b) {
            mbar_expect_tx(bar0 + b * 8, uint32_t(tiles) * kBlockBytes);
            if (!(blockIdx.x == 0 && b == a.fault_block))
                bulk_copy_g2s(smem_u32(blocks + b * kPair), src + b * stride, uint32_t(tiles) * kBlockBytes, bar0 + b * 8);
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int units = a.kb * 2, u0 = units * warp / kTilePairWarps, u1 = units * (warp + 1) / kTilePairWarps;
    bool failed = false;
    struct Unit {
        uint4 ca, cb;            // codes of rows g and g + 8
        uint2 field;
        uint32_t zero;
    };
    auto landed = [&](int u) -> bool {
        if (mbar_wait(bar0 + (u >> 1) * 8, 0, a.wait_limit)) return true;
        if (lane == 0 && a.status) atomicOr(a.status, kStatusCopyTimeout);
        return false;
    };
    auto fetch = [&](int u, int tile, Unit& o) {                 // (of a second tile that does not exist: whatever is there)
        const uint8_t* slot = blocks + (u >> 1) * kPair + tile * kBlockBytes;
        o.ca = *reinterpret_cast<const uint4*>(slot + (u & 1) * 512 + lane * 16);
        o.cb = *reinterpret_cast<const uint4*>(slot + (2 + (u & 1)) * 512 + lane * 16);
        o.field = *reinterpret_cast<const uint2*>(slot + kStepOffset + lane * 8);
        o.zero = slot[kZeroOffset + lane];
    };
    auto decode = [&](const Unit& o, int i, uint32_t (&w)[2][4], const auto& gg, const auto& gh) {
        const uint32_t wa = pick(o.ca, i), wb = pick(o.cb, i);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t ua = wa >> (8 * e), ub = wb >> (8 * e);
            w[e][0] = dq_even(ua, gg); w[e][1] = dq_even(ub, gh);
            w[e][2] = dq_odd(ua, gg); w[e][3] = dq_odd(ub, gh);
        }
    };
    constexpr bool kPlain = STEPS == kStepsPlain;
    auto with_chain = [&](uint32_t fields, auto f) {
        if constexpr (STEPS == kStepsFp16) f(Chain<kChainFp16>{});
        else if (STEPS == kStepsMixed && all_factored(fields)) f(Chain<kChainFactored>{});
        else f(Chain<kChainGeneral>{});
    };
    // The weights are constant; x, the bias and y may belong to the previous kernel until it has completed.
    uint32_t first[4][2][4];
    if (a.overlap) {
        __syncthreads();        // barrier initialisation visible to every waiter
        if (u0 < u1 && !(failed = !landed(u0))) {
            Unit o;
            fetch(u0, 0, o);
            with_chain(o.field.x & o.field.y, [&](auto chain) {
                constexpr int CH = decltype(chain)::value;
                const auto gg = make_group<CH, kPlain>(o.zero & 15u, o.field.x), gh = make_group<CH, kPlain>(o.zero >> 4, o.field.y);
#pragma unroll
                for (int i = 0; i < 4; ++i) decode(o, i, first[i], gg, gh);
            });
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    for (int cc = threadIdx.x; cc < a.kb * 32; cc += kTilePairWarps * 32) {       // x, zeros beyond M and K
        const int k = cc * 8;
        uint8_t* dst = xs + (cc >> 3) * kChunk;
#pragma unroll
        for (int m = 0; m < MT * 8; ++m)
            stage_piece<true>(dst + m * 128 + (((cc ^ m) & 7) << 4), a.x + int64_t(m) * a.ldx + k, m < a.m && k < a.k, k, a.k);
    }
    stage_wait();
    __syncthreads();            // x staged; barrier initialisation visible to every waiter

    float acc[2][2][MT][4];     // [tile][chain]: the products of a unit go to two chains in turn
#pragma unroll
    for (int i = 0; i < 16 * MT; ++i) (&acc[0][0][0][0])[i] = 0.0f;
    auto read_x = [&](int u, int i, uint4 (&xv)[MT]) {
        const uint8_t* chunk = xs + ((u >> 1) * 4 + t) * kChunk + g * 128 + ((((u & 1) * 4 + i) ^ g) << 4);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) xv[mt] = *reinterpret_cast<const uint4*>(chunk + mt * (8 * 128));
    };
    auto multiply = [&](int tile, const uint32_t (&w)[2][4], const uint4 (&xv)[MT]) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                float (&d)[4] = acc[tile][e][mt];
                mma_16816(d, w[e], e ? xv[mt].z : xv[mt].x, e ? xv[mt].w : xv[mt].y, d);
            }
    };
    for (int u = u0; u < u1 && !failed; ++u) {
        const bool ahead = a.overlap && u == u0;                 // the first tile's weights are there already
        if (!ahead && (failed = !landed(u))) break;
        Unit o[2];
        fetch(u, 0, o[0]);
        fetch(u, 1, o[1]);
        with_chain(o[0].field.x & o[0].field.y & o[1].field.x & o[1].field.y, [&](auto chain) {
            constexpr int CH = decltype(chain)::value;
            const auto g0 = make_group<CH, kPlain>(o[0].zero & 15u, o[0].field.x), h0 = make_group<CH, kPlain>(o[0].zero >> 4, o[0].field.y);
            const auto g1 = make_group<CH, kPlain>(o[1].zero & 15u, o[1].field.x), h1 = make_group<CH, kPlain>(o[1].zero >> 4, o[1].field.y);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint4 xv[MT];
                uint32_t w[2][4];
                read_x(u, i, xv);
                if (ahead) {
                    multiply(0, first[i], xv);
                } else {
                    decode(o[0], i, w, g0, h0);
                    multiply(0, w, xv);
                }
                decode(o[1], i, w, g1, h1);
                multiply(1, w, xv);
            }
        });
    }
    if (__syncthreads_or(failed) && threadIdx.x == 0) {
        // A warp gave up: look at every block's barrier once more (bounded), so that nothing lands later
        for (int b = 0; b < a.kb; ++b) {
            bool there = false;
            for (int i = 0; i < 4096 && !there; ++i) there = mbar_try_wait(bar0 + b * 8, 0);
        }
    }
    __syncthreads();
#pragma unroll
    for (int tile = 0; tile < 2; ++tile)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            float (&p)[4] = acc[tile][0][mt], (&q)[4] = acc[tile][1][mt];
            red[((warp * 2 + tile) * MT + mt) * 32 + lane] = make_float4(p[0] + q[0], p[1] + q[1], p[2] + q[2], p[3] + q[3]);
        }
    __syncthreads();
    // thread e adds element e of every warp's sums in warp order (fragment order inside a tile, as in the tile kernel)
    const float* sums = reinterpret_cast<const float*>(red);
    auto sum_of = [&](int e) {
        float sum = 0.0f;
#pragma unroll
        for (int w = 0; w < kTilePairWarps; ++w) sum += sums[w * (2 * MT * 128) + e];
        return sum;
    };
    if (a.act) {
        for (int e = threadIdx.x; e < MT * 128; e += kTilePairWarps * 32) {
            const int tile = e / (MT * 64), r = e % (MT * 64), mt = r >> 6, rl = (r >> 1) & 31, c = r & 1;
            const int at = (tile * MT + mt) * 128 + rl * 4 + c;
            const float gate = sum_of(at), up = sum_of(at + 2);
            const int m = mt * 8 + 2 * (rl & 3) + c, row = nt + tile, n = row * 16 + (rl >> 2);
            if (tile < tiles && m < a.m && n + 8 < a.n)
                a.y[int64_t(m) * a.ldy + row * 8 + (rl >> 2)] = silu_mul(finish_output(gate, a.bias, n), finish_output(up, a.bias, n + 8));
        }
        return;
    }
    for (int e = threadIdx.x; e < 2 * MT * 128; e += kTilePairWarps * 32) {
        const int tile = e / (MT * 128), mt = (e >> 7) % MT, rl = (e >> 2) & 31, c = e & 3;
        const float sum = sum_of(e);
        const int m = mt * 8 + 2 * (rl & 3) + (c & 1), n = (nt + tile) * 16 + (rl >> 2) + 8 * (c >> 1);
        if (tile < tiles && m < a.m && n < a.n) a.y[int64_t(m) * a.ldy + n] = finish_output(sum, a.bias, n);
    }
}

}  // namespace b2
