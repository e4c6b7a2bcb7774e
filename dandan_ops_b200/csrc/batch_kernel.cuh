// Batch kernel: a weight-streaming projection on the 5th-generation tensor cores for up to 128 rows of x.
//
// At these batch sizes every weight is used once per launch, so the work is to fetch the image and to decode it; the
// streaming kernel does that too, but its mma.sync products cost as much again as the decoding from 17 rows of x on
// (eight per fragment at 64 rows).  Here the decoded weights go to tensor memory as the A operand of one
// tcgen05.mma per 16 columns of K, issued by a single thread and the same instruction whatever the number of rows:
//
//   D[n][m] (FP32, tensor memory: 128 lanes = weight rows, NX columns = rows of x; batch_chains() of them, added on reading)
//     += A[n][k] (weights, FP16, tensor memory, written by the converter warps) * B[m][k] (x, shared memory, TMA)
//
// Work split, one of three forms (plan_batch() in batch.cu chooses):
//   ranges    ("stream-K") The layer is cut into steps = (tile of 128 weight rows) x (64 columns of K), numbered tile by tile and
//             dealt out in equal contiguous ranges to one persistent CTA per SM (a block of 256 columns that two CTAs share is
//             fetched and decoded by both, each multiplying its own steps).  A tile that several CTAs share is added up by the
//             last of them to arrive (a ticket per tile and warp, nobody waits), in CTA order, so the result does not depend on
//             which that is.
//   clusters  (CL) A cluster of CTAs (or one CTA) per tile, each with an equal share of the blocks of K.  The sums meet in shared memory: of
//             every four columns of D one CTA is the owner, to which the others send theirs (st.async, counted on its barrier) and
//             which adds them in CTA order.  One trip between SMs instead of store, fence, ticket and load through L2.
//   rounds    More tiles than CTAs: every CTA takes the same number of whole tiles, all CTAs the same columns of K at a time, which
//             streams faster than ranges that begin anywhere.  The tiles left over are shared, each by as many CTAs with an
//             equal share of K as there are, and come first: their sums travel (as those of ranges do) under the products of
//             the whole tiles, and the launch ends with plain stores.
//
// Roles (20 warps):
//   warp 0      bulk copies of the raw blocks: one copy per 256 columns of K (8 native blocks, contiguous)
//   warp 1      issues the MMAs, one wait and one commit per block (256 columns)
//   warp 2      TMA loads of x, one tile of NX rows x 64 columns per step
//   warp 3      allocates and frees tensor memory
//   warps 4..19 converters: two sets of eight warps (two per tensor-memory lane quadrant, two quantization groups each)
//               that take the blocks in turn; they also read the accumulators back, NX / 4 columns each.  A tile's
//               epilogue runs after the warp's first block of a later tile: the tensor cores are through with it by then.
//
// Lane l of quadrant q holds weight row 32q + 16 (l & 1) + 8 hi8 + g of the tile: neighbouring lanes read from two blocks
// and two row pairs, which makes the 16-byte reads of the codes two-way bank conflicts (four-way in row order).
//
// Barriers (bounded waits; a role that gives up raises the CTA's abort flag and the others leave):
//   raw_full/raw_free[r]  bulk copy of a block landed / its converter warps have read it
//   full[b % R]           the x tiles (bytes) and the eight converter warps' weights of block b are in place
//   done[b % R]           tcgen05.commit: the MMAs of block b have completed
//   acc_full/acc_free[b]  accumulator b complete (commit) / read by all converter warps
//   sums                  (CL) the other CTAs' sums have landed (bytes)
#pragma once
#include "gemm_kernel.cuh"

namespace b2 {

constexpr int kBatchRows = 128;                     // weight rows per tile
constexpr int kBatchBlocks = kBatchRows / 16;       // native blocks per 256 columns
constexpr int kBatchRawBytes = kBatchBlocks * kBlockBytes;
constexpr int kBatchEarly = 2;                      // blocks requested ahead of everything else
constexpr uint32_t kBatchWCols = 32;                // tensor-memory columns of a step's weights
constexpr int kBatchSets = 2;                       // sets of eight converter warps (three sets, 72 registers: 3-4 % slower)
constexpr int kBatchWarps = 8 * kBatchSets;
constexpr int kBatchThreads = (4 + kBatchWarps) * 32;
__host__ __device__ constexpr int batch_nx(int64_t m) { return m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128; }    // rows of x of an MMA
enum : int { kRanges = 0, kClusters = 1, kRounds = 2, kDeep = 3 };                  // work splits (kDeep: clusters with sixteen chains)
// Ring of 256-column stages (x tiles in shared memory, weights in tensor memory): what 512 columns leave beside the accumulators.
__host__ __device__ constexpr int batch_ring(int nx, int form) { return form == kRanges ? (nx <= 64 ? 3 : 2) : nx == 16 && form != kDeep ? 3 : 2; }
// The FP32 sums of a tile run as C chains (the products of 16 columns of K go to chain kk % C), added in order when they
// are read: a tensor core drops the bits of a product below the running sum, so the error grows with the length of a
// chain.  Share of FP16 outputs that are not the nearest to the 64-bit sum, one chain -> four or two (streaming kernel / K-split GEMM):
// 4096 x 12288 at M = 16 1.4 % -> 0.4 % (0.6 %), M = 24 1.4 -> 0.5 (0.7), M = 64 1.4 -> 0.8 (0.75); 6144 x 4096 at M = 16
// 0.7 -> 0.2 (0.4).  Ranges, whose CTAs have more than one tile, have as many as fit beside the weight ring, and a second accumulator
// where that leaves four chains.  The other forms, which share a tile among fewer CTAs, have twice as many, in place of the second
// accumulator (up to 16 rows) or of a stage of the ring: 6144 x 4096 at M = 24 / 64 0.21 / 0.37 % as ranges of three CTAs per tile, in clusters
// of two 0.29 / 0.53 with the chains of the ranges, 0.17 / 0.30 with twice as many (7.75 -> 7.94, 9.14 -> 9.31 us; the most it costs is 8192 x
// 28672 at M = 64 42.2 -> 48.2, ranges 48).  Up to 16 rows sixteen instead of eight where the tile kernel would take the layer, whose
// chains have two to four products (kDeep: 2048 x 5120 at M = 8 0.09 %, tile kernel 0.09, eight chains 0.12; 4.78, 5.96 and 4.39 us).
__host__ __device__ constexpr int batch_chains(int nx, int form) {
    return form == kRanges ? (nx <= 32 ? 4 : 2) : nx == 16 && form != kDeep ? 8 : 256 / nx;
}
__host__ __device__ constexpr int batch_accs(int nx, int form) { return nx == 16 && form == kRanges ? 2 : 1; }
__host__ __device__ constexpr int batch_x_bytes(int nx) { return nx * 128; }          // 64 columns
// Sums a CTA of a cluster receives: from every other one, of the units (four columns x 128 weight rows) that it owns.
constexpr int kBatchUnitBytes = kBatchRows * 16;
__host__ __device__ constexpr int batch_sums_bytes(int nx, int c) { return (c - 1) * ((nx / 4 + c - 1) / c) * kBatchUnitBytes; }
// Cluster sizes in use; what they need beside the rings.  With 128 rows of x there is no room left, and the sums go to the x tiles
// (which no CTA of the cluster may still be reading then, see `ready` in the kernel).
constexpr int kBatchClusters[] = {2, 3, 4, 6, 8};
__host__ __device__ constexpr int batch_sums_area(int nx, int form) {
    int most = 0;
    for (int c : kBatchClusters) most = batch_sums_bytes(nx, c) > most ? batch_sums_bytes(nx, c) : most;
    return (form == kClusters || form == kDeep) && nx <= 64 ? most : 0;
}
__host__ __device__ constexpr int batch_raw_stages(int nx, int form) {
    const int fit = (232448 - 1024 - 512 - 4 * batch_ring(nx, form) * batch_x_bytes(nx) - batch_sums_area(nx, form)) / kBatchRawBytes;
    return fit < 8 ? fit : 8;
}
__host__ __device__ constexpr int batch_smem_bytes(int nx, int form) {
    return 1024 + 4 * batch_ring(nx, form) * batch_x_bytes(nx) + batch_raw_stages(nx, form) * kBatchRawBytes + batch_sums_area(nx, form) + 512;
}
// Bytes of all partial tiles of a launch: a CTA has at most two tiles that it shares.
__host__ __device__ constexpr int64_t batch_partial_bytes(int nx, int grid) { return int64_t(grid) * 2 * nx * kBatchRows * 4; }

struct BatchArgs {
    const uint8_t* native;
    __half* y;
    const __half* bias;     // optional [N] FP16 (may be null)
    float4* partial;        // [CTA][first or last tile][NX / 4][128 weight rows] x 4 columns
    unsigned* tickets;      // [CTA][warp], zero on entry and on exit
    unsigned* status;
    int64_t ldy;
    int m, n;
    int n16, kb;
    int steps;              // tiles * kb * 4 (ranges)
    int shared_tiles, whole;    // tiles that several CTAs share, and that every CTA takes by itself (rounds)
    int cluster, parts;     // CTAs per tile (clusters), per shared tile (rounds); their blocks of K: kb_each, the first kb_more of them one more
    int kb_each, kb_more;
    int row_tiles;          // tiles of NX rows of x (MANY)
    int act;                // as StreamArgs::act
    int wait_limit;
    int fault_block;        // -1; a test passes b >= 0: CTA 0 arms the barrier of its b-th block but skips the copy
};

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// CW columns of this thread's lane (4 or 8), complete after tcgen05.wait::ld.
template <int CW>
__device__ __forceinline__ void batch_ld(uint32_t taddr, uint32_t (&v)[CW]) {
    static_assert(CW == 4 || CW == 8, "4 or 8 columns");
    if constexpr (CW == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(taddr) : "memory");
}
// The sums of CW accumulator columns: the C chains (NX columns apart), G of them requested before a wait, added in a fixed order.
// (G = 4 where the converters' loop follows: with eight it spilled, 24576 x 4096 at M = 16 18.0 -> 18.7 us.)
template <int NX, int C, int CW, int G = C>
__device__ __forceinline__ void batch_sums(uint32_t taddr, float (&f)[CW]) {
    constexpr int W = CW < 8 || G >= 8 ? 4 : 8;
#pragma unroll
    for (int at = 0; at < CW; at += W)
#pragma unroll
        for (int c0 = 0; c0 < C; c0 += G) {
            uint32_t v[G][W];
#pragma unroll
            for (int c = 0; c < G; ++c) batch_ld<W>(taddr + (c0 + c) * NX + at, v[c]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < G; ++c)
#pragma unroll
                for (int i = 0; i < W; ++i) {
                    asm volatile("" : "+r"(v[c][i]));                              // (not used before the wait)
                    f[at + i] = c0 + c == 0 ? __uint_as_float(v[c][i]) : __fadd_rn(f[at + i], __uint_as_float(v[c][i]));
                }
        }
}

// First step of CTA c's range, and the CTA whose range contains step s.
// (32-bit: steps * ctas stays below 2^32, see batch_applicable; 64-bit divisions took 0.4 us of a launch.)
__device__ __forceinline__ int batch_begin(int steps, int ctas, int c) { return int(unsigned(steps) * unsigned(c) / unsigned(ctas)); }
__device__ __forceinline__ int batch_owner(int s, int steps, int ctas) { return int((unsigned(s + 1) * unsigned(ctas) - 1u) / unsigned(steps)); }

__device__ __forceinline__ uint32_t peer_address(uint32_t own, int rank) {                // the same place in another CTA of the cluster
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(own), "r"(rank));
    return r;
}

// MANY: x has more than NX rows.  A tile is then NX rows of x by 128 weight rows, numbered with the rows of x inside, so that CTAs side by
// side read the same weights.
template <int NX, int STEPS, int FORM, bool MANY = false>
__global__ void __launch_bounds__(kBatchThreads, 1)
w4a16_batch_kernel(const __grid_constant__ CUtensorMap xmap, const BatchArgs a) {
    constexpr bool CL = FORM == kClusters || FORM == kDeep;
    constexpr int R = batch_ring(NX, FORM), RS = batch_raw_stages(NX, FORM), kXBytes = batch_x_bytes(NX), kXStage = 4 * kXBytes;
    constexpr uint32_t kWStage = 4 * kBatchWCols, kWBase = 512 - R * kWStage;
    constexpr int C = batch_chains(NX, FORM), ACCS = batch_accs(NX, FORM);
    static_assert(ACCS * C * NX <= int(kWBase) && RS >= 4, "tensor memory and shared memory hold the rings");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* x_base = smem;                                                // [R][4][kXBytes]
    uint8_t* raw_base = x_base + R * kXStage;                              // [RS][18688]
    uint8_t* sums = NX <= 64 ? raw_base + RS * kBatchRawBytes : x_base;    // (CL) [other CTA][unit of this one][weight row] x 4 columns
    uint64_t* bars = reinterpret_cast<uint64_t*>(raw_base + RS * kBatchRawBytes + batch_sums_area(NX, FORM));
    constexpr int RAW_FULL = 0, RAW_FREE = RAW_FULL + RS, FULL = RAW_FREE + RS, DONE = FULL + R, ACC_FULL = DONE + R,
                  ACC_FREE = ACC_FULL + 2, DRAIN = ACC_FREE + 2, SUMS = DRAIN + 1, NBARS = SUMS + 1;
    static_assert(NBARS * 8 + 8 <= 512, "barrier area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NBARS);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + i * 8; };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ctas = gridDim.x;
    const int tsteps = a.kb * 4;                                           // steps of a tile
    int rank = 0, tile0, kb0, b0 = 0, nsteps = 0, nblocks;                 // first tile and block; range of steps; blocks of 8 x 256 columns
    int nshared = 0;                                                       // (rounds) blocks of a shared tile, before the whole ones
    if constexpr (CL) {                                                    // whole blocks of one tile, without a division
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%clusterid.x;" : "=r"(tile0));
        kb0 = rank * a.kb_each + min(rank, a.kb_more);
        nblocks = a.kb_each + (rank < a.kb_more ? 1 : 0);
    } else if constexpr (FORM == kRounds) {
        tile0 = int(blockIdx.x) / a.parts;
        rank = int(blockIdx.x) - tile0 * a.parts;
        kb0 = rank * a.kb_each + min(rank, a.kb_more);
        if (tile0 < a.shared_tiles) {
            nshared = a.kb_each + (rank < a.kb_more ? 1 : 0);
        } else {
            tile0 = a.shared_tiles + int(blockIdx.x);
            kb0 = 0;
        }
        nblocks = nshared + a.whole * a.kb;
    } else {
        b0 = batch_begin(a.steps, ctas, blockIdx.x);
        nsteps = batch_begin(a.steps, ctas, blockIdx.x + 1) - b0;
        nblocks = ((b0 + nsteps - 1) >> 2) - (b0 >> 2) + 1;
        tile0 = (b0 >> 2) / a.kb;
        kb0 = (b0 >> 2) - tile0 * a.kb;
    }
    auto weight_tile = [&](int tile) { return MANY ? tile / a.row_tiles : tile; };
    auto first_row = [&](int tile) { return MANY ? tile % a.row_tiles * NX : 0; };          // of x
    int tile = tile0, kb = kb0;                                            // (warps 0 and 2: of the block at hand)
    auto next_block = [&](int b) {                                         // from block b - 1 to b
        if (FORM == kRounds && b == nshared) {
            tile = a.shared_tiles + int(blockIdx.x);
            kb = 0;
        } else if (++kb == a.kb) {
            kb = 0;
            tile += FORM == kRounds ? ctas : 1;
        }
    };
    const int first_end = FORM == kRounds && nshared ? nshared : a.kb - kb0;                // blocks up to the end of the first tile

    auto request = [&](int b, int tile, int kb) {                           // block b of the range
        const int r = b % RS;
        const uint32_t bytes = uint32_t(min(kBatchBlocks, a.n16 - tile * kBatchBlocks)) * kBlockBytes;
        mbar_expect_tx(bar(RAW_FULL + r), bytes);
        if (!(blockIdx.x == 0 && b == a.fault_block))
            bulk_copy_g2s(smem_u32(raw_base + r * kBatchRawBytes),
                          a.native + (int64_t(kb) * a.n16 + tile * kBatchBlocks) * kBlockBytes, bytes, bar(RAW_FULL + r));
    };
    // The first blocks are on their way before anything else happens: their trip is the longest part of the start.  (Not a
    // whole ring of them: x would queue up behind all CTAs' rings.)
    int issued = 0;                                                        // (warp 0: next block to request)
    if (warp == 0) {
        static_assert(RS <= 32 && NBARS - RS <= 32, "a lane per barrier");
        if (lane < RS) mbar_init(bar(RAW_FULL + lane), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        for (; issued < min(kBatchEarly, nblocks); ++issued) {
            if (elect_one()) request(issued, weight_tile(tile), kb);
            __syncwarp();
            next_block(issued + 1);
        }
        if (const int i = RAW_FREE + lane; i < NBARS)
            mbar_init(bar(i), i < FULL ? 8 : i < DONE ? 1 + 8 : i >= ACC_FREE && i < DRAIN ? kBatchWarps : 1);
        if (lane == 0) *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        if (elect_one()) {
            if constexpr (CL) {
                const int units = (min(a.m - first_row(tile0), NX) + 3) / 4;        // in use; this CTA owns every a.cluster-th
                mbar_expect_tx(bar(SUMS), uint32_t((a.cluster - 1) * ((units - rank + a.cluster - 1) / a.cluster) * kBatchUnitBytes));
            }
        }
        __syncwarp();
    }
    if (warp == 2 && elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    // Phases of the cluster barrier, the same in every thread: `ready` - the others may write to this CTA's `sums` - and
    // `sent` - this thread writes to nobody any more; a CTA leaves only when all threads of its cluster have got that far.
    auto cluster_arrive = [] { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); };
    auto cluster_wait = [] { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); };
    if (warp == 3) tmem_alloc(smem_u32(tmem_slot), 512);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if constexpr (CL && NX <= 64) cluster_arrive();                        // `sums` has a place of its own: ready from the start

    // Bounded; the lanes of a warp go on or leave together.  As a programmatic dependent the kernel may have been held up by
    // the one before it, which can last longer than the limit (a gather that waits for its peers): a limit that has run
    // out counts once more from that kernel's end.  (The same wait up front in every role cost 1 % of small launches.)
    auto wait = [&](int idx, uint32_t parity) -> bool {
        const uint32_t at = bar(idx);
        if (__all_sync(0xffffffffu, mbar_try_wait(at, parity))) return true;
        for (int turn = 0; turn < 2; ++turn) {
            for (int i = 1; i < a.wait_limit; ++i) {
                if (__all_sync(0xffffffffu, mbar_try_wait_long(at, parity))) return true;
                if ((i & 63) == 63 && __any_sync(0xffffffffu, *abort_flag != 0)) return false;
            }
            if (turn == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
        }
        if (lane == 0) {
            *abort_flag = 1;
            atomicOr(a.status, kStatusGemmTimeout);
        }
        return false;
    };

    if (warp == 0) {
        // ------------------------------ raw blocks ---------------------------------------
        for (; issued < nblocks; ++issued) {
            const int r = issued % RS;
            if (issued >= RS && !wait(RAW_FREE + r, ((issued / RS) - 1) & 1)) break;
            if (elect_one()) request(issued, weight_tile(tile), kb);
            __syncwarp();
            next_block(issued + 1);
        }
        // after an abort: the last copies land before the shared memory is released
        for (int i = max(0, issued - RS); i < issued; ++i)
            for (int p = 0; p < 4096 && !mbar_try_wait(bar(RAW_FULL + i % RS), (i / RS) & 1); ++p) {}
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ---------------------------------------
        // D = F32, A = B = F16, both K-major, M = 128 weight rows, N = NX rows of x
        const uint32_t idesc = (1u << 4) | (uint32_t(NX >> 3) << 17) | (uint32_t(kBatchRows >> 4) << 24);
        const uint64_t desc0 = umma_desc_sw128(smem_u32(x_base));
        int left = first_end;                         // blocks to the end of the tile
        int seg = 0;
        bool fresh = true;                            // the accumulator starts with this block
        bool ok = true;
        for (int b = 0; b < nblocks; ++b) {
            const int slot = b % R;
            if (fresh && seg >= ACCS && !(ok = wait(ACC_FREE + seg % ACCS, (seg / ACCS - 1) & 1))) break;
            if (!(ok = wait(FULL + slot, (b / R) & 1))) break;
            tcgen05_fence_after();
            const bool end = --left == 0 || b == nblocks - 1;
            if (elect_one()) {
                const uint32_t w = tmem_base + kWBase + slot * kWStage, d = tmem_base + seg % ACCS * (C * NX);
                const uint64_t desc = desc0 + uint64_t((slot * kXStage) >> 4);
                uint32_t accumulate = fresh ? 0u : 1u;
                auto step = [&](int t) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const int i = t * 4 + kk;                     // (ranges, which may begin inside a block, have four chains at most)
                        umma_f16_ts(d + i % C * NX, w + t * kBatchWCols + kk * 8, desc + uint64_t((t * kXBytes) >> 4) + uint64_t(kk * 2), idesc,
                                    (C > 4 ? i : kk) < C ? accumulate : 1u);
                    }
                    if (C <= 4) accumulate = 1;
                };
                const int t0 = FORM == kRanges && b == 0 ? b0 & 3 : 0;                                      // steps of the range in this block
                const int t1 = FORM == kRanges && b == nblocks - 1 ? (b0 + nsteps - 1) & 3 : 3;
                if (t0 == 0 && t1 == 3) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) step(t);
                } else {
#pragma unroll 1
                    for (int t = t0; t <= t1; ++t) step(t);
                }
                umma_commit(bar(DONE + slot));
                if (end) umma_commit(bar(ACC_FULL + seg % ACCS));
            }
            __syncwarp();
            fresh = end;
            if (end) {
                ++seg;
                left = a.kb;
            }
        }
        if (!ok) {                                    // after an abort: MMAs in flight end before their operands are released
            if (elect_one()) umma_commit(bar(DRAIN));
            __syncwarp();
            for (int p = 0; p < 4096 && !mbar_try_wait(bar(DRAIN), 0); ++p) {}
        }
    } else if (warp == 2) {
        // ------------------------------ x tiles ------------------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int b = 0; b < nblocks; ++b) {
            const int slot = b % R;
            if (b >= R && !wait(DONE + slot, ((b / R) - 1) & 1)) break;
            if (elect_one()) {
                const int t0 = FORM == kRanges && b == 0 ? b0 & 3 : 0, t1 = FORM == kRanges && b == nblocks - 1 ? (b0 + nsteps - 1) & 3 : 3;
                mbar_expect_tx(bar(FULL + slot), uint32_t(t1 - t0 + 1) * kXBytes);
                for (int t = t0; t <= t1; ++t)
                    tma_load_2d(smem_u32(x_base + slot * kXStage + t * kXBytes), &xmap, (kb * 4 + t) * kGemmBK, first_row(tile), bar(FULL + slot));
            }
            __syncwarp();
            next_block(b + 1);
        }
    } else if (warp >= 4) {
        // ------------------------------ converters ---------------------------------------
        const int quad = warp & 3, u = (warp - 4) >> 2, v = u & 1, set = u >> 1;
        const int blk = lane & 1, hi8 = (lane >> 2) & 1, g = ((lane >> 1) & 1) | ((lane >> 3) << 1);
        const int row = quad * 32 + blk * 16 + hi8 * 8 + g;                // weight row of the tile
        const uint32_t lane_addr = uint32_t(quad * 32) << 16;
        const int code_at = (quad * 2 + blk) * kBlockBytes + (2 * hi8) * 512 + (4 * g + 2 * v) * 16;
        const int step_at = (quad * 2 + blk) * kBlockBytes + kStepOffset + (4 * g + 2 * v) * 8 + hi8 * 4;
        const int zero_at = (quad * 2 + blk) * kBlockBytes + kZeroOffset + 4 * g + 2 * v;
        constexpr int CW = NX >= 64 ? 16 : NX / 4;                         // accumulator columns per read
        bool ok = true;
        int read = 0;                                                      // tiles of the range that this warp has read

        // The sums of this lane's weight row and the rows m0.. of x -> y.
        auto emit = [&](int tile, int m0, const auto& f) {
            constexpr int W = sizeof(f) / sizeof(float);
            const int n = weight_tile(tile) * kBatchRows + row, base = first_row(tile), rows = a.m - base;
            __half* y = a.y + int64_t(base) * a.ldy;
            if (a.act) {
                // lanes l and l ^ 4 hold the gate and the up sum of one output column: the gate lane
                // finishes the even rows of x, the up lane the odd ones
                const int out = (n >> 4) * 8 + g;
#pragma unroll
                for (int i = 0; i < W; i += 2) {
                    const float theirs = __shfl_xor_sync(0xffffffffu, hi8 ? f[i] : f[i + 1], 4);
                    const float gate = hi8 ? theirs : f[i], up = hi8 ? f[i + 1] : theirs;
                    const int m = m0 + i + hi8;
                    if (m < rows && (n | 8) < a.n)
                        y[int64_t(m) * a.ldy + out] = silu_mul(finish_output(gate, a.bias, n & ~8), finish_output(up, a.bias, n | 8));
                }
            } else if (n < a.n) {
#pragma unroll
                for (int i = 0; i < W; ++i)
                    if (m0 + i < rows) y[int64_t(m0 + i) * a.ldy + n] = finish_output(f[i], a.bias, n);
            }
        };

        // A tile that other CTAs share, in three steps: partial sums out, ticket drawn, and, if it was the last, all sums read back.
        // Rounds take a block of the next tile between them, so that none waits for the one before.
        int pending = 0, shared_tile = 0, first = 0, last = 0;              // steps done, of which tile, and its CTAs
        unsigned prior = 0;
        auto slot_of = [&](int c) {                                        // partial tile of CTA c, this warp's columns and lanes
            return a.partial + ((int64_t(c) * 2 + (c == first ? 1 : 0)) * (NX / 4) + u * (NX / 16)) * kBatchRows + quad * 32 + lane;
        };
        auto draw_ticket = [&] {
            __threadfence();
            __syncwarp();
            unsigned* ticket = a.tickets + first * kBatchWarps + (warp - 4);
            if (lane == 0) {
                prior = atomicAdd(ticket, 1u);
                if (prior == unsigned(last - first)) *ticket = 0u;
            }
            pending = 2;
        };
        auto read_back = [&] {
            pending = 0;
            if (__shfl_sync(0xffffffffu, prior, 0) != unsigned(last - first)) return;
            __threadfence();
            const int rows = a.m - first_row(shared_tile);
            constexpr int RW = CW < 8 ? CW : 8, PARTS = 32 / RW;           // partial tiles requested together, added in CTA order
#pragma unroll 1
            for (int c0 = 0; c0 < NX / 4; c0 += RW) {
                const int m0 = u * (NX / 4) + c0;
                if (m0 >= rows) break;
                float f[RW];
#pragma unroll
                for (int i = 0; i < RW; ++i) f[i] = 0.0f;
                for (int c = first; c <= last; c += PARTS) {
                    float4 p[PARTS][RW / 4];
#pragma unroll
                    for (int j = 0; j < PARTS; ++j)
#pragma unroll
                        for (int q = 0; q < RW / 4; ++q)
                            if (c + j <= last && m0 + 4 * q < rows) p[j][q] = __ldcg(slot_of(c + j) + (c0 / 4 + q) * kBatchRows);
                            else p[j][q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int j = 0; j < PARTS; ++j)
#pragma unroll
                        for (int q = 0; q < RW / 4; ++q) {
                            f[4 * q] += p[j][q].x; f[4 * q + 1] += p[j][q].y; f[4 * q + 2] += p[j][q].z; f[4 * q + 3] += p[j][q].w;
                        }
                }
                emit(shared_tile, m0, f);
            }
        };
        auto advance = [&] {
            if (pending == 1) draw_ticket();
            else if (pending == 2) read_back();
        };
        auto epilogue = [&](int seg) {
            const int tile = FORM == kRounds ? (seg == 0 ? tile0 : a.shared_tiles + int(blockIdx.x) + (seg - (nshared ? 1 : 0)) * ctas) : tile0 + seg;
            if (seg == 0) asm volatile("griddepcontrol.wait;" ::: "memory");   // bias, tickets, partial tiles, y
            ok = ok && wait(ACC_FULL + seg % ACCS, (seg / ACCS) & 1);
            if (!ok) return;
            tcgen05_fence_after();
            bool whole;
            if constexpr (FORM == kRounds) {
                whole = seg > 0 || nshared == 0 || a.parts == 1;
                if (!whole) {                                              // (a whole tile may be read while a shared one is pending)
                    first = tile * a.parts;
                    last = first + a.parts - 1;
                }
            } else {
                const int t0 = tile * tsteps, t1 = t0 + tsteps;
                whole = b0 <= t0 && t1 <= b0 + nsteps;
                first = whole ? 0 : batch_owner(t0, a.steps, ctas);
                last = whole ? 0 : batch_owner(t1 - 1, a.steps, ctas);
            }
            const uint32_t acc = tmem_base + lane_addr + seg % ACCS * (C * NX) + u * (NX / 4);
            const int rows = a.m - first_row(tile);
            if (whole) {
#pragma unroll
                for (int c0 = 0; c0 < NX / 4; c0 += CW) {
                    const int m0 = u * (NX / 4) + c0;
                    if (m0 < rows) {
                        float f[CW];
                        batch_sums<NX, C, CW, (C > 4 ? 4 : C)>(acc + c0, f);
                        emit(tile, m0, f);
                    }
                }
            } else {
                float4* dst = slot_of(int(blockIdx.x));
#pragma unroll
                for (int c0 = 0; c0 < NX / 4; c0 += CW) {
                    float f[CW];
                    batch_sums<NX, C, CW, (C > 4 ? 4 : C)>(acc + c0, f);
#pragma unroll
                    for (int q = 0; q < CW / 4; ++q)
                        if (u * (NX / 4) + c0 + 4 * q < rows)
                            __stcg(dst + (c0 / 4 + q) * kBatchRows, make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]));
                }
                pending = 1;
                shared_tile = tile;
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(ACC_FREE + seg % ACCS));
            if (FORM == kRanges && !whole) {
                draw_ticket();
                read_back();
            }
        };

        // Clusters: unit U (columns 4U..4U + 3) belongs to CTA U % cluster, as its unit U / cluster.
        auto exchange = [&] {
            ok = ok && wait(ACC_FULL, 0);
            if (ok) tcgen05_fence_after();
            __syncwarp();
            if constexpr (NX > 64) cluster_arrive();                       // all products of this CTA are done: nothing reads its x tiles
            cluster_wait();
            constexpr int kUnits = NX / 16;                                // of this warp
            const int rows = a.m - first_row(tile0);
            const int c = a.cluster, own_units = (NX / 4 + c - 1) / c, inverse = 65536 / c + 1;      // U / c for U < 32
            const uint32_t lane_at = uint32_t(quad * 32 + lane) * 16, acc0 = tmem_base + lane_addr + u * (NX / 4);
            float f[NX / 4];
            if (ok) {
#pragma unroll
                for (int c0 = 0; c0 < NX / 4; c0 += CW)
                    if (u * (NX / 4) + c0 < rows) {
                        float (&mine)[CW] = *reinterpret_cast<float (*)[CW]>(f + c0);
                        batch_sums<NX, C, CW>(acc0 + c0, mine);
#pragma unroll
                        for (int q = 0; q < CW / 4; ++q) {
                            const int U = u * kUnits + c0 / 4 + q, i = U * inverse >> 16, owner = U - i * c;
                            if (owner == rank || 4 * U >= rows) continue;
                            const int from = rank < owner ? rank : rank - 1;
                            send_sums(peer_address(smem_u32(sums) + (from * own_units + i) * kBatchUnitBytes + lane_at, owner),
                                      make_float4(mine[4 * q], mine[4 * q + 1], mine[4 * q + 2], mine[4 * q + 3]), peer_address(bar(SUMS), owner));
                        }
                    }
            }
            __syncwarp();
            cluster_arrive();                                              // sent
            if (!ok) return;
            asm volatile("griddepcontrol.wait;" ::: "memory");             // bias, y
            if (!(ok = wait(SUMS, 0))) return;
#pragma unroll
            for (int q = 0; q < kUnits; ++q) {
                const int U = u * kUnits + q, i = U * inverse >> 16;
                if (U - i * c != rank || 4 * U >= rows) continue;
                float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
                for (int r = 0; r < c; ++r) {                              // in CTA order
                    float4 p = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
                    if (r != rank) p = *reinterpret_cast<const float4*>(sums + ((r < rank ? r : r - 1) * own_units + i) * kBatchUnitBytes + lane_at);
                    t[0] += p.x; t[1] += p.y; t[2] += p.z; t[3] += p.w;
                }
                emit(tile0, 4 * U, t);
            }
        };

        int slot = set, r = set, b = set;                                  // rings, and the warp's block
        uint32_t free_parity = 1, raw_parity = 0;                          // (the first round of the stages is free)
        // Up to and with the first block behind the oldest tile that has not been read (`tile_end`): its products are in the making
        // while that tile is read.
        int tile_end = first_end;
        while (ok && b < nblocks) {
            const int stop = CL ? nblocks : min(nblocks, FORM == kRounds && pending ? b + kBatchSets : tile_end + kBatchSets);
            for (; b < stop; b += kBatchSets) {
                if (!(ok = wait(RAW_FULL + r, raw_parity))) break;
                const uint8_t* raw = raw_base + r * kBatchRawBytes;
                const uint4 code[4] = {*reinterpret_cast<const uint4*>(raw + code_at), *reinterpret_cast<const uint4*>(raw + code_at + 512),
                                       *reinterpret_cast<const uint4*>(raw + code_at + 16), *reinterpret_cast<const uint4*>(raw + code_at + 528)};
                const uint32_t fields[2] = {*reinterpret_cast<const uint32_t*>(raw + step_at), *reinterpret_cast<const uint32_t*>(raw + step_at + 8)};
                const uint32_t zeros = *reinterpret_cast<const uint16_t*>(raw + zero_at) >> (4 * hi8);
                auto convert = [&](int h, auto chain) {
                    const auto gc = make_group<decltype(chain)::value, STEPS == kStepsPlain>((zeros >> (8 * h)) & 15u, fields[h]);
                    const uint32_t words[8] = {code[2 * h].x, code[2 * h].y, code[2 * h].z, code[2 * h].w,
                                               code[2 * h + 1].x, code[2 * h + 1].y, code[2 * h + 1].z, code[2 * h + 1].w};
                    const uint32_t to = tmem_base + lane_addr + kWBase + slot * kWStage + (2 * v + h) * kBatchWCols;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 p = dequant_word(words[2 * i], gc), q = dequant_word(words[2 * i + 1], gc);
                        if (h == 0 && i == 0) {
                            if (!(ok = wait(DONE + slot, free_parity))) return;
                            tcgen05_fence_after();
                        }
                        tmem_st8(to + 8 * i, p, q);
                    }
                };
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if constexpr (STEPS == kStepsFp16) convert(h, Chain<kChainFp16>{});
                    else if (STEPS == kStepsMixed && all_factored(fields[h])) convert(h, Chain<kChainFactored>{});
                    else convert(h, Chain<kChainGeneral>{});
                    if (!ok) break;
                }
                if (!ok) break;
                tmem_st_wait();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bar(FULL + slot));
                    if (b + RS < nblocks) mbar_arrive(bar(RAW_FREE + r));      // the last copies are not waited for
                }
                if ((slot += kBatchSets) >= R) { slot -= R; free_parity ^= 1; }
                if ((r += kBatchSets) >= RS) { r -= RS; raw_parity ^= 1; }
            }
            if constexpr (!CL) {
                if (FORM == kRounds && pending) advance();
                for (; ok && tile_end <= b - kBatchSets; tile_end += a.kb) epilogue(read++);
            }
        }
        if constexpr (CL) {
            exchange();
        } else {
            const int segs = FORM == kRounds ? a.whole + (nshared ? 1 : 0) : (b0 + nsteps - 1) / tsteps - tile0 + 1;
            while (read < segs && ok) epilogue(read++);
            if constexpr (FORM == kRounds)
                while (pending) advance();
        }
    }
    __syncwarp();
    if constexpr (CL) {
        if (warp < 4) {                                // (the converters have been through these)
            if constexpr (NX > 64) cluster_arrive();
            cluster_wait();
            cluster_arrive();
        }
        cluster_wait();                                // nobody writes to this CTA any more
    }
    tcgen05_fence_before();
    __syncthreads();
    // After an abort x tiles may be on their way to stages whose barrier the converters never completed, and sums of other CTAs
    // to a place that this one does not wait for: whoever gave up, all roles have stopped requesting, and the last loads and
    // stores get 0.1 ms to land.
    for (int p = 0; p < 64 && *abort_flag; ++p) __nanosleep(2000);
    if (warp == 3) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace b2
