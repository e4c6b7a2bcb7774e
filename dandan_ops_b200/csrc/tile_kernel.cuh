// Latency-oriented kernel for small and mid-size layers in the decode regime (M <= 16).
//
// On layers of a few megabytes the streaming kernel is bound by latency, not bandwidth: a
// warp needs ~0.5 us to decode one native block, and splitting K between CTAs costs a trip
// through global memory.  This kernel puts the whole K range of one row tile (16 outputs)
// into one CTA and brings every one of its native blocks in flight at once:
//   * one bulk copy and one mbarrier per native block, all issued by the first thread before
//     anything else happens (kb * 2336 bytes in flight per CTA, several CTAs per SM);
//   * the unit of work is half a block (eight of its sixteen MMA steps); up to 16 warps take
//     consecutive units, so a block is decoded by two warps in parallel;
//   * as a programmatic dependent a warp decodes its first unit before it waits for the previous kernel of the stream (up to
//     8 rows of x; 4096 x 1024 at M = 1 / 8 in a chain of launches 3.3 / 3.4 -> 2.7 / 2.8 us, 6144 x 1024 3.4 / 3.6 -> 3.0 / 3.1;
//     64 registers, so that two CTAs of 16 warps share an SM);
//   * x for the CTA's K range is staged once, unpadded: rows of 128 bytes per 64-column chunk
//     with the 16-byte pieces XOR-swizzled by the row, so the fragment reads are conflict-free
//     and two CTAs of a 4096-column layer share an SM at M = 8;
//   * the per-warp FP32 accumulator tiles are added in warp order through shared memory, so
//     the result is bit-reproducible and no workspace, ticket or partial tile is needed;
//   * layers with few row tiles and a long K run a cluster of 2 or 4 CTAs per row tile, each
//     on its share of K; the sums of CTAs 1.. are sent to CTA 0's shared memory (st.async, counted on a barrier there).
// The dequantization chain and the MMA fragment layout are those of stream_kernel.cuh.
#pragma once
#include <type_traits>
#include "layout.cuh"
#include "stream_kernel.cuh"

namespace b2 {

constexpr int kTileMaxWarps = 16;

struct TileArgs {
    const __half* x;
    const uint8_t* native;
    __half* y;
    unsigned* status;       // may be null
    const __half* bias;     // optional [N] FP16 (may be null)
    int64_t ldx, ldy;
    int m, n, k;
    int n16, kb;
    int warps;              // warps per CTA = min(16, 2*kb)
    int act;                // as StreamArgs::act
    int wait_limit;         // mbarrier polls before a warp gives up (a test passes a small number)
    int fault_block;        // -1; a test passes b >= 0: CTA 0 arms the barrier of its b-th block but skips the copy
    int ksplit;             // 1, 2 or 4: a cluster of that many CTAs shares a row tile, each takes its share
                            // of the K blocks and the others send their 16 x 8*MT sums to the first one's shared
                            // memory (layers whose row tiles leave most SMs idle)
    int overlap;            // launched as a programmatic dependent of the previous kernel: all weight copies are
                            // requested first, then the kernel waits for that one before it reads x
};

// `rows` = rows of x that exist (1..16): only those are staged, so that at M = 1 a CTA of a
// 4096-column layer needs 55 KB instead of 120 KB and four of them share an SM.
// Staged x: per 64-column chunk `rows` rows of 128 bytes, the eight 16-byte pieces of row m stored at
// piece index p ^ (m & 7), chunks 32 bytes apart modulo 128: the 16-byte fragment reads of a quarter
// warp (two rows, four chunks) fall into eight different bank groups without padding the rows.
__host__ __device__ constexpr int tile_x_chunk_bytes(int rows) { return rows * 128 + 32; }
__host__ __device__ constexpr int tile_smem_bytes(int kb, int rows, int warps) {
    // barriers (padded to 128) + blocks + staged x + reduction tiles
    return ((kb * 8 + 127) / 128) * 128 + kb * kBlockBytes + kb * 4 * tile_x_chunk_bytes(rows) +
           warps * (rows <= 8 ? 1 : 2) * 512;
}

// Element e of a row tile's 16 x (8 * MT) sums (fragment order: e = mt * 128 + 4 * lane + c) -> one output.
// GATHER: threads e and e ^ 16 hold neighbouring columns of the same row; they exchange their values so that
// the even one has a 4-byte word, which it stores into the local buffer and sends to every peer's mailbox.
// Every lane of a warp must call this in the same iteration (the callers' loops guarantee it).
template <bool GATHER>
__device__ __forceinline__ void tile_emit(const TileArgs& a, const GatherArgs* ga, int nt, int e, float sum) {
    const int mt = e >> 7, rl = (e >> 2) & 31, c = e & 3;
    const int rg = rl >> 2, rt = rl & 3;
    const int m = mt * 8 + 2 * rt + (c & 1), n = nt * 16 + rg + 8 * (c >> 1);
    const bool inside = m < a.m && n < a.n;
    if constexpr (!GATHER) {
        if (inside) a.y[int64_t(m) * a.ldy + n] = finish_output(sum, a.bias, n);
    } else {
        const unsigned v = inside ? unsigned(__half_as_ushort(finish_output(sum, a.bias, n))) : 0u;
        const unsigned other = __shfl_xor_sync(0xffffffffu, v, 16);          // column n ^ 1 of the same row
        if ((rg & 1) == 0 && inside) {
            const unsigned word = v | (other << 16);
            *reinterpret_cast<unsigned*>(a.y + int64_t(m) * a.ldy + n) = word;
            const unsigned epoch = mailbox_epoch(*ga);
            const int64_t s = int64_t(m) * (ga->cols >> 1) + (n >> 1);
            for (int q = 0; q < ga->world; ++q)
                if (q != ga->rank)
                    mailbox_send(mailbox(ga->flags[q], ga->world, ga->slots, epoch & 1u, ga->rank) + s, word, epoch);
        }
    }
}

// End of a writer CTA in the gather form: count it; the last one of the grid's n16 writers collects the peers'
// packets with all its threads and publishes the epoch.
__device__ __forceinline__ void tile_collect(const TileArgs& a, const GatherArgs* ga) {
    __shared__ int last;
    unsigned* mine = ga->flags[ga->rank];
    const unsigned epoch = mailbox_epoch(*ga);                   // read before this CTA counts itself
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(mine + kGatherTicketWord, 1u) == unsigned(a.n16) - 1u;
    __syncthreads();
    if (!last) return;
    if (mailbox_receive(*ga, epoch, threadIdx.x, blockDim.x)) atomicOr(mine + kGatherStatusWord, kStatusPeerTimeout);
    __syncthreads();
    if (threadIdx.x == 0) {
        mine[kGatherEpochWord] = epoch;
        mine[kGatherTicketWord] = 0u;
    }
}

// The warps' tiles added in warp order, for the fragment at `red` of the first warp's.
template <int MT>
__device__ __forceinline__ float4 tile_sum(const float4* red, int warps) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int w = 0; w < warps; ++w) {
        const float4 f = red[w * (MT * 32)];
        v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
    }
    return v;
}

// FULL: all MT * 8 rows of x are staged (zeros beyond M): compile-time layout, no row predicates -
// the faster form whenever the padded rows do not cost occupancy.  Otherwise only the M rows that
// exist are staged and lanes of missing rows use zero fragments.
//
// GATHER: the multi-GPU form (b2_w4a16_linear_gather).  `a.y` is this rank's column slice of a full [M, N]
// buffer; the CTA that writes a row tile stores it there and sends it to every peer's mailbox as
// {word, epoch} packets (tile_emit).  The grid of this kernel need not be resident at once, so no CTA may wait
// for a peer while others are still to be scheduled: the CTAs count themselves on the flag block's ticket
// when their tile is out, and only the LAST one - by then every packet of this rank has left - collects the
// packets the peers sent (bounded as everywhere) and publishes the epoch.
//
// SPLIT: a cluster of a.ksplit CTAs per row tile (always FULL: those grids are small).  A kernel of its own, so that layers of one CTA
// per tile do not carry it: 6144 x 1024 at M = 1 / 4 3.00 / 3.08 -> 2.71 / 2.95 us, a chain of 3072 x 2048, 2048 x 2048, 8192 x 2048 and
// 2048 x 4096 16.4 / 16.8 -> 15.2 / 16.2.  (A chain that takes both in turn starts each with cold instructions: the projections of a
// 0.6B layer 11.1 against 11.2 in one kernel at M = 1, 12.0 against 11.9 at M = 4.)
template <int MT, bool XVEC, bool FULL, int STEPS, bool GATHER, bool SPLIT>
__device__ __forceinline__ void tile_body(const TileArgs& a, const GatherArgs* ga) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int rows = FULL ? MT * 8 : a.m;
    const int ksplit = SPLIT ? a.ksplit : 1;
    const int kChunk = tile_x_chunk_bytes(rows);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    // this CTA's share of the row tile: blocks kb0 .. kb0 + kbn - 1 of K
    uint32_t part = 0;
    if (ksplit > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(part));
    const int nt = blockIdx.x / ksplit;
    const int kb0 = int(part) * a.kb / ksplit, kbn = (int(part) + 1) * a.kb / ksplit - kb0;
    const int kb_max = (a.kb + ksplit - 1) / ksplit;     // all CTAs of a cluster use one layout
    const int bar_bytes = ((kb_max * 8 + 127) / 128) * 128;
    uint8_t* blocks = smem + bar_bytes;
    uint8_t* xs = blocks + kb_max * kBlockBytes;
    float4* red = reinterpret_cast<float4*>(xs + kb_max * 4 * kChunk);
    const uint32_t bar0 = smem_u32(smem);

    auto sums_bar = [&] { return smem_u32(red + a.warps * MT * 32); };       // (clusters) behind the reduction tiles
    if (threadIdx.x == 0) {
        for (int b = 0; b < kbn; ++b) mbar_init(bar0 + b * 8, 1);
        if (!GATHER && ksplit > 1 && part == 0) mbar_init(sums_bar(), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!GATHER && ksplit > 1 && part == 0) mbar_expect_tx(sums_bar(), uint32_t(ksplit - 1) * (MT * 512));
        const uint8_t* src = a.native + (int64_t(kb0) * a.n16 + nt) * kBlockBytes;
        const int64_t stride = int64_t(a.n16) * kBlockBytes;
        for (int b = 0; b < kbn; ++b) {
            mbar_expect_tx(bar0 + b * 8, kBlockBytes);
            if (!(blockIdx.x == 0 && b == a.fault_block))
                bulk_copy_g2s(smem_u32(blocks + b * kBlockBytes), src + b * stride, kBlockBytes, bar0 + b * 8);
        }
    }
    if (ksplit > 1) {
        // First phase of "every CTA of the cluster runs and the first one's barrier for the sums is set up", completed before the
        // hand-over below touches another CTA's shared memory: thread 0 arrives behind its initialisation, made visible to the cluster
        // by the fence.  (Nobody waits for this phase until its products are done.)
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    }
    // Kernels launched behind this one as programmatic dependents may start as soon as they find room.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // units = half blocks, dealt in consecutive runs to the warps
    const int units = kbn * 2;
    const int u0 = (units * warp) / a.warps, u1 = (units * (warp + 1)) / a.warps;
    bool failed = false;
    // Codes, step fields and zero points of the lane's two rows in half h of block b, and the fragments of word i of them.
    struct Unit {
        uint4 ca, cb;
        uint2 field;
        uint32_t zero;
    };
    // A lane that gives up a wait goes on with whatever is in the block: products and votes are instructions of the whole warp, and the
    // other lanes may have seen the copy land.  (A vote behind the wait costs 1024 x 2048 at M = 1 / 8 5 / 1 %, 6144 x 1024 1 / 0; where
    // K is split at 9 to 16 rows it gains 3.)
    constexpr bool kVote = SPLIT && MT == 2;
    auto await = [&](uint32_t barrier) {
        if constexpr (kVote) {
            if (failed || mbar_wait(barrier, 0, a.wait_limit)) return;
        } else {
            if (mbar_try_wait(barrier, 0)) return;
            for (int i = failed ? a.wait_limit : 1; i < a.wait_limit; ++i)
                if (mbar_try_wait_long(barrier, 0)) return;
        }
        if (!failed && a.status) atomicOr(a.status, kStatusCopyTimeout);
        failed = true;
    };
    auto fetch = [&](int u, Unit& o) {
        const int b = u >> 1, h = u & 1;
        await(bar0 + b * 8);
        const uint8_t* slot = blocks + b * kBlockBytes;
        o.ca = *reinterpret_cast<const uint4*>(slot + h * 512 + lane * 16);           // row g
        o.cb = *reinterpret_cast<const uint4*>(slot + (2 + h) * 512 + lane * 16);     // row g+8
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
    auto with_chain = [&](const Unit& o, auto f) {
        auto go = [&](auto chain) {
            constexpr int CH = decltype(chain)::value;
            constexpr bool kPlain = STEPS == kStepsPlain;
            f(make_group<CH, kPlain>(o.zero & 15u, o.field.x), make_group<CH, kPlain>(o.zero >> 4, o.field.y));
        };
        if constexpr (STEPS == kStepsFp16) go(Chain<kChainFp16>{});
        else if (STEPS == kStepsMixed && all_factored(o.field.x & o.field.y)) go(Chain<kChainFactored>{});
        else go(Chain<kChainGeneral>{});
    };
    // The weights are constant; x, the bias and y may belong to the previous kernel until it has completed.  With one row tile
    // of x (registers) a warp decodes its first unit meanwhile.
    constexpr bool kAhead = MT == 1;
    uint32_t first[kAhead ? 4 : 1][2][4];
    if constexpr (kAhead) {
        if (a.overlap) {
            __syncthreads();        // barrier initialisation visible to every waiter
            Unit o;
            if (u0 < u1) {
                fetch(u0, o);
                with_chain(o, [&](const auto& gg, const auto& gh) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) decode(o, i, first[i], gg, gh);
                });
            }
        }
    }
    if (a.overlap) asm volatile("griddepcontrol.wait;" ::: "memory");
    // stage x for all columns (zero beyond M and K)
    {
        // Copies that bypass registers (cp.async) are the faster form for the small grids of a K split
        // (2 %), loads through registers for grids that fill the device (6144 x 1024: 4.5 vs 5.2 us).
        auto stage = [&](auto async) {
            constexpr bool kAsync = decltype(async)::value;
            const int pieces_per_row = kbn * 32;
            for (int cc = threadIdx.x; cc < pieces_per_row; cc += blockDim.x) {
                const int k = kb0 * kBlockCols + cc * 8;
                uint8_t* dst = xs + (cc >> 3) * kChunk;
                const __half* src = a.x + k;
                if constexpr (FULL) {
#pragma unroll
                    for (int m = 0; m < MT * 8; ++m)
                        stage_piece<XVEC, kAsync>(dst + m * 128 + (((cc ^ m) & 7) << 4), src + int64_t(m) * a.ldx,
                                                  m < a.m && k < a.k, k, a.k);
                } else {
                    for (int m = 0; m < rows; ++m)
                        stage_piece<XVEC, kAsync>(dst + m * 128 + (((cc ^ m) & 7) << 4), src + int64_t(m) * a.ldx,
                                                  k < a.k, k, a.k);
                }
            }
            if constexpr (XVEC && kAsync) stage_wait();
        };
        if (ksplit > 1) stage(std::true_type{}); else stage(std::false_type{});
    }
    __syncthreads();        // x staged; barrier initialisation visible to every waiter

    // The eight MMAs of a unit would be one dependent chain per row tile of x; kChains accumulator tiles used in
    // turn cut it into chains of 8 / kChains (four at one row tile, two at two), added in a fixed order at the end.
    constexpr int kChains = MT == 1 ? 4 : 2;
    float acc[MT][4], accx[kChains - 1][MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            acc[mt][c] = 0.0f;
#pragma unroll
            for (int q = 0; q < kChains - 1; ++q) accx[q][mt][c] = 0.0f;
        }
    auto multiply = [&](int u, int i, const uint32_t (&w)[2][4]) {
        const int b = u >> 1, h = u & 1;
        const uint8_t* xchunk = xs + (b * 4 + t) * kChunk + g * 128;
        uint4 xv[MT];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)      // rows of x that do not exist are not staged: their columns of the product are zero
            xv[mt] = (FULL || mt * 8 + g < rows) ? *reinterpret_cast<const uint4*>(xchunk + mt * (8 * 128) + (((h * 4 + i) ^ g) << 4))
                                                 : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int chain = (kChains == 4 ? 2 * (i & 1) + e : e);       // compile-time under the unrolling
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                float (&dst)[4] = chain == 0 ? acc[mt] : accx[chain == 0 ? 0 : chain - 1][mt];
                mma_16816(dst, w[e], e ? xv[mt].z : xv[mt].x, e ? xv[mt].w : xv[mt].y, dst);
            }
        }
    };
    int u = u0;
    if constexpr (kAhead) {
        if (a.overlap && u0 < u1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) multiply(u0, i, first[i]);
            ++u;
        }
    }
    for (; u < u1; ++u) {
        Unit o;
        fetch(u, o);
        with_chain(o, [&](const auto& gg, const auto& gh) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t w[2][4];
                decode(o, i, w, gg, gh);
                multiply(u, i, w);
            }
        });
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int q = 0; q < kChains - 1; ++q) acc[mt][c] += accx[q][mt][c];
    // Blocks this CTA requested but no warp waited for cannot exist: every block has two units.
    if (__syncthreads_or(failed) && threadIdx.x == 0) {
        // A warp gave up: copies of this CTA may still be in flight.  Look at every block's barrier
        // once more (bounded) so that nothing lands in shared memory after the CTA has left.
        for (int b = 0; b < kbn; ++b) {
            bool landed = false;
            for (int i = 0; i < 4096 && !landed; ++i) landed = mbar_try_wait(bar0 + b * 8, 0);
        }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
        red[(warp * MT + mt) * 32 + lane] = make_float4(acc[mt][0], acc[mt][1], acc[mt][2], acc[mt][3]);
    __syncthreads();
    if constexpr (SPLIT && !GATHER) {
        // The CTAs of a cluster share the row tile.  Each adds its warps' tiles in warp order; the others send their sums to the
        // first one's shared memory, counted on its barrier, and it adds them to its own in CTA order and writes y.  (Against plain
        // remote stores between two cluster barriers 1024 x 2048 at M = 1 / 8 / 16 2.74 / 2.98 / 3.97 -> 2.47 / 2.75 / 3.66 us.)
        const float4* peer = red + (a.warps + 1) * MT * 32;                // [ksplit - 1][MT * 32] the others' sums
        const bool adds = threadIdx.x < MT * 32;                           // a thread per fragment of the sums
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (adds) v = tile_sum<MT>(red + threadIdx.x, a.warps);
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");        // CTA 0 runs, its barrier is set up
        if (adds && part != 0) {
            uint32_t to, bar;
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(smem_u32(peer + (part - 1) * (MT * 32) + threadIdx.x)));
            asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(bar) : "r"(sums_bar()));
            send_sums(to, v, bar);
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // this thread sends nothing any more
        if (adds && part == 0) {
            const bool landed = mbar_wait(sums_bar(), 0, a.wait_limit);
            if (landed) {
                for (int p = 0; p + 1 < ksplit; ++p) {
                    const float4 f = peer[p * (MT * 32) + threadIdx.x];
                    v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
                }
                const int m = int(threadIdx.x >> 5) * 8 + 2 * t, n = nt * 16 + g;
                if (a.act) {                                               // gate (row g) and up (row g + 8) of two rows of x
                    if (n + 8 < a.n) {
                        if (m < a.m) a.y[int64_t(m) * a.ldy + nt * 8 + g] = silu_mul(finish_output(v.x, a.bias, n), finish_output(v.z, a.bias, n + 8));
                        if (m + 1 < a.m) a.y[int64_t(m + 1) * a.ldy + nt * 8 + g] = silu_mul(finish_output(v.y, a.bias, n), finish_output(v.w, a.bias, n + 8));
                    }
                } else {
                    __half* y = a.y + int64_t(m) * a.ldy + n;
                    if (m < a.m && n < a.n) y[0] = finish_output(v.x, a.bias, n);
                    if (m + 1 < a.m && n < a.n) y[a.ldy] = finish_output(v.y, a.bias, n);
                    if (m < a.m && n + 8 < a.n) y[8] = finish_output(v.z, a.bias, n + 8);
                    if (m + 1 < a.m && n + 8 < a.n) y[a.ldy + 8] = finish_output(v.w, a.bias, n + 8);
                }
            } else if (lane == 0 && a.status) {
                atomicOr(a.status, kStatusCopyTimeout);
            }
            failed = !landed;
        }
        __syncwarp();
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");        // nobody writes to this CTA any more
        if (__syncthreads_or(failed)) __nanosleep(100000);                 // (but for sums that were on their way when it gave up)
        return;
    }
    if (GATHER && SPLIT && ksplit > 1) {
        // The gather form, by plain stores between two cluster barriers: each CTA adds its warps' tiles in warp order; CTA p > 0 puts its
        // 128 * MT sums into slot p - 1 of the first one's shared memory, and after the cluster barrier the first adds the slots to its
        // own sums in CTA order and writes y.
        float* tot = reinterpret_cast<float*>(red) + a.warps * MT * 128;       // [MT * 128] own sums
        float* peer = tot + MT * 128;                                          // [ksplit - 1][MT * 128] the others' sums
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        for (int e = threadIdx.x; e < MT * 128; e += blockDim.x) {
            const int mt = e >> 7, rl = (e >> 2) & 31, c = e & 3;
            float sum = 0.0f;
            for (int w = 0; w < a.warps; ++w)
                sum += reinterpret_cast<const float*>(red)[((w * MT + mt) * 32 + rl) * 4 + c];
            if (part == 0) {
                tot[e] = sum;
            } else {
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(smem_u32(peer + (part - 1) * (MT * 128) + e)));
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(sum) : "memory");
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (part != 0) return;
        for (int e = threadIdx.x; e < MT * 128; e += blockDim.x) {
            float sum = tot[e];
            for (int p = 0; p + 1 < ksplit; ++p) sum += peer[p * (MT * 128) + e];
            tile_emit<GATHER>(a, ga, nt, e, sum);
        }
        if constexpr (GATHER) tile_collect(a, ga);
        return;
    }
    // thread e adds element e of every warp's tile in warp order and stores one output
    if (a.act) {
        // gate (row rg) and up (row rg + 8) of one output: elements c and c + 2 of the same fragment
        for (int e = threadIdx.x; e < MT * 64; e += blockDim.x) {
            const int mt = e >> 6, rl = (e >> 1) & 31, c = e & 1;
            float gate = 0.0f, up = 0.0f;
            for (int w = 0; w < a.warps; ++w) {
                const float* f = reinterpret_cast<const float*>(red) + ((w * MT + mt) * 32 + rl) * 4;
                gate += f[c];
                up += f[c + 2];
            }
            const int rg = rl >> 2, rt = rl & 3;
            const int m = mt * 8 + 2 * rt + c, n = nt * 16 + rg;
            if (m < a.m && n + 8 < a.n)
                a.y[int64_t(m) * a.ldy + nt * 8 + rg] = silu_mul(finish_output(gate, a.bias, n), finish_output(up, a.bias, n + 8));
        }
        return;
    }
    for (int e = threadIdx.x; e < MT * 128; e += blockDim.x) {
        const int mt = e >> 7, rl = (e >> 2) & 31, c = e & 3;
        float sum = 0.0f;
        for (int w = 0; w < a.warps; ++w)
            sum += reinterpret_cast<const float*>(red)[((w * MT + mt) * 32 + rl) * 4 + c];
        tile_emit<GATHER>(a, ga, nt, e, sum);
    }
    if constexpr (GATHER) tile_collect(a, ga);
}

template <int MT, bool XVEC, bool FULL, int STEPS = kStepsMixed, bool SPLIT = false>
__global__ void __launch_bounds__(kTileMaxWarps * 32, 2)
w4a16_tile_kernel(const TileArgs a) {
    tile_body<MT, XVEC, FULL, STEPS, false, SPLIT>(a, nullptr);
}

template <int MT, bool FULL, int STEPS>
__global__ void __launch_bounds__(kTileMaxWarps * 32, 2)
w4a16_tile_gather_kernel(const TileArgs a, const GatherArgs ga) {
    tile_body<MT, true, FULL, STEPS, true, FULL>(a, &ga);
}

}  // namespace b2
