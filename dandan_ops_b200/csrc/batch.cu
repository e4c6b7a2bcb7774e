// Launch plan and launch of the batch kernel (batch_kernel.cuh).
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <climits>

#include "../../include/b2_w4a16.h"
#include "batch.cuh"
#include "host_common.cuh"

namespace {

// Estimated time of a launch beyond its fixed start, in ns: the longest range of steps, the shared tiles in it (store, fence and
// ticket of each), and the reading of a tile's partial sums by the last CTA (measured on per-CTA time stamps).
int launch_cost(int nx, int steps, int tsteps, int grid) {
    const int range = (steps + grid - 1) / grid;
    const int tiles = steps / tsteps;
    const bool aligned = grid % tiles == 0;                     // every CTA inside one tile
    const int parts = aligned ? grid / tiles : (tsteps + range - 1) / range + 1;
    const int step_ns = nx <= 32 ? 220 : nx == 64 ? 250 : 310;
    return range * step_ns + (parts == 1 ? 0 : (aligned ? 1 : 2) * 1300 + parts * (200 + 7 * nx));
}

constexpr int kRangeBlocks = 11, kRangeBlocksCluster = 8;   // blocks of K that equal ranges must gain per SM to pay for their hand-over
constexpr int kMaxPerTile = 16;      // CTAs per tile looked at: beyond, the partial sums cost more than the shorter ranges give

// Clusters of c CTAs of the kernel that a device of so many SMs runs at the same time: those of a B200 (what
// cudaOccupancyMaxActiveClusters() says of its 148 SMs), in proportion.  Not asked of the device at hand: which of its SMs are there
// differs from one to the next, and the plan, and with it the order of the sums, must not.  (A cluster that finds no place waits for one.)
int cluster_capacity(int c, int sms) {
    static constexpr int kB200[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    return kB200[c] * sms / 148;
}

}  // namespace

namespace b2host {

// Estimated time of a launch with c CTAs per tile (one: whole tiles, no sums to send) beyond its fixed start, in ns: the blocks of a
// CTA, and, the more SMs a launch takes, the later the next one finds room to start under it.  Fitted to 33 layers of 512 x 1024
// to 9216 x 4096 at 1 to 128 rows in chains of launches, all cluster sizes measured: off by 2 to 6 % (rms), the chosen size
// 0.7 % slower than the fastest in the mean.
int cluster_cost(int nx, int tiles, int kb, int c) {
    const int block_ns = nx <= 32 ? 455 : nx == 64 ? 525 : 750, exchange_ns = nx == 16 ? 350 : nx == 32 ? 700 : nx == 64 ? 1100 : 1400;
    const int blocks = (kb + c - 1) / c, ctas = tiles * c;
    return blocks * block_ns + ctas * (2000 + 85 * blocks) / 148 + (c > 1 ? exchange_ns : 0);
}

// Time that the tiles left over by whole rounds take, in ns, if each is shared by `parts` CTAs: their blocks, the slower the more
// of the SMs are at it, and the trip of the partial sums.  Fitted to 54 layers of 149 to 592 tiles and K = 512 to 8192 at 16 to 128
// rows, every number of CTAs measured: off by 5 % of a launch (rms), the chosen number 1 % slower than the fastest in the mean.
int shared_cost(int nx, int tiles, int kb, int parts, int sms) {
    const int alone_ns = nx <= 32 ? 290 : nx == 64 ? 350 : 670, crowd_ns = nx <= 32 ? 435 : nx == 64 ? 500 : 630;
    const int share_ns = nx <= 32 ? 1400 : nx == 64 ? 2200 : 2600, part_ns = nx == 16 ? 0 : nx == 32 ? 30 : nx == 64 ? 110 : 270;
    return (kb + parts - 1) / parts * (alone_ns + crowd_ns * tiles * parts / sms) + (parts > 1 ? share_ns + part_ns * parts : 0);
}

BatchPlan plan_batch(int64_t m, const b2::Dims& d, int sm_count) {
    BatchPlan p;
    p.nx = b2::batch_nx(m);
    p.row_tiles = int((m + p.nx - 1) / p.nx);
    p.cluster = p.parts = 1;
    p.whole = p.shared_tiles = 0;
    p.deep = false;
    const int tiles = (d.n + b2::kBatchRows - 1) / b2::kBatchRows * p.row_tiles, tsteps = d.kb * 4;
    const int64_t steps = int64_t(tiles) * tsteps;
    p.steps = int(steps);
    // Ranges: equal ones over all SMs, or the same number of CTAs for every tile (shorter hand-over, a few SMs idle).
    const int device_sms = sm_count > 0 ? sm_count : 148, sms = int(std::min<int64_t>(device_sms, steps));
    int best_cost = launch_cost(p.nx, p.steps, tsteps, sms);
    p.grid = sms;
    for (int g = tiles; g <= std::min(sms, kMaxPerTile * tiles); g += tiles) {
        const int cost = launch_cost(p.nx, p.steps, tsteps, g);
        if (cost <= best_cost) { best_cost = cost; p.grid = g; }
    }
    const int64_t range = (steps + p.grid - 1) / p.grid;
    p.max_parts = p.grid % tiles == 0 ? p.grid / tiles : int(std::min<int64_t>(p.grid, (tsteps + range - 1) / range + 1));
    p.partial_bytes = b2::batch_partial_bytes(p.nx, p.grid);
    // A tensor core's error grows with the products that a chain of sums takes: a CTA of the other forms, which have twice the chains of
    // the ranges up to 64 rows and as many above, may have no more of them than the ranges would.  (6144 x 4096 at M = 128 in 96 CTAs
    // 13.1 us, in 144 as ranges 14.8, 0.53 against 0.37 % of the outputs not the nearest.)
    const int chains = b2::batch_chains(p.nx, b2::kClusters) / b2::batch_chains(p.nx, b2::kRanges);
    auto short_chains = [&](int blocks) { return p.row_tiles > 1 || blocks * 4 <= range * chains; };
    bool one_round = false;
    if (tiles >= sms && (p.row_tiles > 1 || chains > 1)) {
        // Rounds, us with ranges / rounds at M = 16, 32 and 64: 28672 x 1024 11.4 / 7.6, 12.6 / 8.8, 14.6 / 10.0, 24576 x 4096 20.0 / 18.0, 21.4 / 20.0,
        // 23.8 / 22.2, 57344 x 8192 70.2 / 65.0, 77.5 / 76.2, level.  Not at 128 rows, whose rounds would have longer chains (24576 x 4096 37.2
        // against 34.4 us then).
        p.grid = sms;
        p.whole = tiles / sms;
        p.shared_tiles = tiles % sms;
        int best = INT_MAX;
        for (int parts = 1; p.shared_tiles && parts <= std::min({kMaxPerTile, sms / p.shared_tiles, d.kb}); ++parts) {
            const int cost = shared_cost(p.nx, p.shared_tiles, d.kb, parts, sms);
            if (cost < best) { best = cost; p.parts = parts; }
        }
        p.max_parts = p.parts;
        // Where few SMs have a last tile and K is long, ranges after all: 28672 x 8192 at M = 16 39.3 against 37.3, 30720 x 8192 level.
        const int blocks = p.whole * d.kb + (p.shared_tiles ? (d.kb + p.parts - 1) / p.parts : 0);
        if (int64_t(blocks) * sms - int64_t(tiles) * d.kb > int64_t(kRangeBlocks) * sms) {
            p.whole = p.shared_tiles = 0;
            p.parts = 1;
            p.max_parts = int(std::min<int64_t>(p.grid, (tsteps + range - 1) / range + 1));
        }
    } else if (tiles <= cluster_capacity(2, device_sms)) {
        // A layer whose tiles all find a cluster at the same time (74 of two CTAs on a B200) takes one, or one CTA, per tile: us with the
        // better ranges / the cluster, at M = 1, 16, 64 and 128: 6144 x 4096 (two CTAs) 8.3 / 6.7, 8.8 / 7.0, 11.5 / 9.3, ranges; 4096 x 12288
        // (four) 11.3 / 9.8, 11.8 / 10.2, 15.1 / 12.3, 22.1 / 16.6; 1024 x 4096 (eight) 3.3 / 3.1, 4.8 / 4.1, 9.9 / 5.7, 14.4 / 8.4; 8192 x 8192 (two)
        // at M = 32 and 64 16.0 / 13.6, 17.2 / 14.6, with K = 28672 40.6 / 38.5, level.
        // Sizes above two leave a cluster free (5760 x 12288 with all 45 clusters of three at M = 16 14.3 -> 15.6).  Where so few CTAs per
        // tile fit that many SMs idle, ranges over all of them win on the longest K: 6144 x 28672 at M = 16 26.8 against 31.2, 6144 x
        // 12288 16.8 against 17.5; 7168 x 16384 23.2 against 21.6.
        int best = INT_MAX, c = 0;
        for (const int size : {1, 2, 3, 4, 6, 8}) {
            if (d.kb < size || tiles > cluster_capacity(size, device_sms) - (size > 2 ? 1 : 0) || !short_chains((d.kb + size - 1) / size)) continue;
            const int cost = cluster_cost(p.nx, tiles, d.kb, size);
            if (cost < best) { best = cost; c = size; }
        }
        if (c && ((d.kb + c - 1) / c) * (sms - tiles * c) <= (c > 1 ? kRangeBlocksCluster : kRangeBlocks) * sms) {
            p.cluster = p.max_parts = c;
            p.grid = tiles * c;
            one_round = c == 1;
        }
    } else if (tiles < sms) {
        // One whole tile per CTA as long as what the other SMs could have taken off them is little: ranges / whole tiles at M = 16, 76 x 128
        // columns with K = 4096 14.1 / 12.1, 5120 15.2 / 15.5, 8192 18.5 / 20.2, 97 x 128 with 5120 15.3 / 13.7, 8192 20.5 / 20.8, 12288 26.3 / 28.9.
        one_round = d.kb * (sms - tiles) <= kRangeBlocks * sms && short_chains(d.kb);
    }
    if (one_round) {
        p.grid = tiles;
        p.max_parts = 1;
        // (of the shortest K as a range per tile: two accumulators or a longer ring; 6144 x 1024 at M = 32 4.3 us, as a round 4.75)
        p.whole = p.nx != 32 || d.kb >= 8 || d.kb * 4 > range ? 1 : 0;
    }
    // Sixteen chains where the tile kernel, whose chains have two to four products, would be the next best.
    const int64_t blocks = int64_t(d.n16) * d.kb;
    const bool tile = m > 8 ? blocks <= (d.kb <= 12 ? 2304 : 4096) : blocks <= (d.n < 4096 ? 8192 : 4096);
    p.deep = p.nx == 16 && (p.cluster > 1 || one_round) && tile;
    // (up to 128 rows a smaller workspace than that of the ranges is refused whatever the form)
    if (p.row_tiles > 1 && (p.cluster > 1 || p.max_parts == 1)) p.partial_bytes = 0;
    return p;
}

int launch_batch(const BatchPlan& p, const CUtensorMap& xmap, const b2::BatchArgs& a, int steps, bool overlap, cudaStream_t s) {
    if (p.row_tiles > 1) return launch_batch_row_tiles(p, xmap, a, steps, overlap, s);
    if (p.cluster > 1 || p.deep) return launch_batch_clusters(p, xmap, a, steps, overlap, s);
    return p.whole ? launch_batch_rounds(p, xmap, a, steps, overlap, s) : launch_batch_ranges(p, xmap, a, steps, overlap, s);
}

}  // namespace b2host
