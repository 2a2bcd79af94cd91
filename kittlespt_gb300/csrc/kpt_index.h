// kpt_index.h -- the kernels' index arithmetic that reaches the end of a
// 32-bit range, also as plain C++ (tests/index_range.cpp walks it on the CPU).
#pragma once

#ifdef __CUDACC__
#define KPT_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define KPT_HOST_DEVICE inline
#endif

namespace kpt {

// use(i, whether it is the lane that stores) for every i in [i0, n) that
// `thread` of a grid of `threads` (whole warps) takes, LANES neighbouring lanes
// to an i.  With several, whole warps: the groups past the end repeat the last.
// Unsigned: i < 2^31 and, where a grid of one thread per i covers n, a stride
// of up to 2^31, whose sum an int does not hold from n = 2^30 + 1 on.
template <int LANES, class Use>
KPT_HOST_DEVICE void spread(unsigned thread, unsigned threads, int i0, int n, Use use) {
    const unsigned all = threads / LANES, end = (unsigned)n;
    if (LANES == 1) {
        for (unsigned i = (unsigned)i0 + thread; i < end; i += all) use((int)i, true);
    } else {
        const unsigned lane = thread & 31u, group = lane / LANES;
        for (unsigned i = (unsigned)i0 + (thread & ~31u) / LANES; i < end; i += all) {   // the warp's first
            const unsigned k = i + group;
            use((int)(k < end ? k : end - 1u), k < end && (lane & (LANES - 1)) == 0);
        }
    }
}

// Lanes of each of `warps` that take rays of a queue of n > 0 rays.
KPT_HOST_DEVICE int lanes_of_queue(int n, int warps) { return (n - 1) / warps + 1; }

// The queue's entry `rank` after the fetch counter's value `base`, and whether
// the queue of n has it.  Unsigned: the counter ends up to a grid's lanes past
// n, beyond 2^31 - 1 for the longest queues.
KPT_HOST_DEVICE int queue_entry(int base, int rank) { return (int)((unsigned)base + (unsigned)rank); }
KPT_HOST_DEVICE bool queued(int entry, int n) { return (unsigned)entry < (unsigned)n; }

// The node (of nn < 2^31) that a thread of a block of block_size threads works
// on where 16 neighbouring threads take one; the thread's number in the grid
// would pass 2^31 - 1 at 2^27 nodes.
KPT_HOST_DEVICE unsigned node_of_16(unsigned block, unsigned block_size, unsigned thread) {
    return block * (block_size / 16u) + thread / 16u;
}

}  // namespace kpt
