// The all-gather of small slices through mailboxes, a launch of its own (gather_kernel.cuh has the parts that projections carry too).
#pragma once
#include "gather_kernel.cuh"

namespace b2 {

static __global__ void __launch_bounds__(256)
gather_mailbox_kernel(const GatherArgs a) {
    const unsigned epoch = mailbox_epoch(a);
    const unsigned parity = epoch & 1u;
    const __half* y = a.y[a.rank];
    const int64_t stride = int64_t(gridDim.x) * blockDim.x, first = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    // ---- send: every word of my slice to every peer's mailbox --------------------------------------
    {
        const int64_t wpr = a.cols >> 1;                                  // 4-byte words per row of my slice
        const int64_t words = int64_t(a.m) * wpr;
        const int peers = a.world - 1;
        for (int64_t i = first; i < words * peers; i += stride) {
            const int pi = int(i / words);
            const int64_t s = i - pi * words;
            const int64_t row = s / wpr, w = s - row * wpr;
            const unsigned data = *reinterpret_cast<const unsigned*>(y + row * a.ld + a.col0 + 2 * w);
            mailbox_send(mailbox(a.flags[pi < a.rank ? pi : pi + 1], a.world, a.slots, parity, a.rank) + s, data, epoch);
        }
    }
    // ---- receive: poll the packets of every peer's slice and copy the words into my buffer ---------
    mailbox_finish(a, epoch, mailbox_receive(a, epoch, first, stride));
}

}  // namespace b2
