// Walks the kernels' index arithmetic (kpt_index.h) at the ends of its ranges.
// Prints "<name> <places checked> <wrong>".
#include <cstdio>
#include <initializer_list>

#include "kpt_index.h"

// k_sky's launch for n directions, blocks of 64 threads: every thread of the
// blocks around the ends and the middle of the grid, and around n - 2^30 and
// 2^31 - (grid), where a signed sum of index and stride changes sign.
template <int LANES>
static void sky(long long n, long long& places, long long& wrong) {
    constexpr long long BLOCK = 64;
    const long long per_block = BLOCK / LANES, blocks = (n - 1) / per_block + 1, threads = blocks * BLOCK;
    for (long long near : {0LL, threads / 3, threads / 2, threads, n - (1LL << 30), (1LL << 31) - threads, (1LL << 30)}) {
        for (long long t = near - 256; t < near + 256; ++t) {
            if (t < 0 || t >= threads) continue;
            int visits = 0, stored = -1;
            bool inside = true;
            kpt::spread<LANES>((unsigned)t, (unsigned)threads, 0, (int)n, [&](int i, bool first) {
                inside = inside && i >= 0 && i < n;
                if (first) stored = i;
                ++visits;
            });
            const long long mine = t / LANES;   // the grid covers n once
            const bool stores = t % LANES == 0 && mine < n;
            const bool warp_in = (t & ~31LL) / LANES < n;
            ++places;
            if (!inside || visits != (warp_in && (LANES > 1 || mine < n) ? 1 : 0) || stored != (stores ? (int)mine : -1)) ++wrong;
        }
    }
}

// A queue of n rays on `warps`: the lanes that take rays (some, and enough for a
// short queue), and the entries at the counter's values around and past n.
static void queue(long long n, int warps, long long& places, long long& wrong) {
    const long long lanes = kpt::lanes_of_queue((int)n, warps);
    ++places;
    if (lanes < 1 || lanes * warps < n || (lanes - 1) * warps >= n) ++wrong;
    for (long long c = n > 40 ? n - 40 : 0; c < n + 32LL * warps; ++c) {
        const int entry = kpt::queue_entry((int)(unsigned)(c - c % 32), (int)(c % 32));
        ++places;
        if (kpt::queued(entry, (int)n) != (c < n) || (c < n && entry != c)) ++wrong;
    }
}

// k_refit_leaves' launch for nn nodes: blocks of 64 threads, 16 to a node.
static void refit(long long nn, long long& places, long long& wrong) {
    constexpr int BLOCK = 64;
    const long long blocks = (nn - 1) / (BLOCK / 16) + 1;
    for (long long near : {0LL, (1LL << 25), (1LL << 26), blocks / 2, blocks})
        for (long long b = near - 3; b < near + 3; ++b)
            for (int t = 0; t < BLOCK && b >= 0 && b < blocks; ++t) {
                const unsigned node = kpt::node_of_16((unsigned)b, BLOCK, (unsigned)t);
                const long long want = (b * BLOCK + t) / 16;
                ++places;
                if ((long long)node != want || (node < (unsigned)nn) != (want < nn)) ++wrong;
            }
}

int main() {
    long long places = 0, wrong = 0;
    for (long long n : {1LL, 31LL, 63LL, 64LL, 65LL, 131072LL, (1LL << 30) - 1, 1LL << 30, (1LL << 30) + 1, 1500000000LL,
                        (1LL << 31) - 65, (1LL << 31) - 64, (1LL << 31) - 63, (1LL << 31) - 1})
        sky<1>(n, places, wrong);
    for (long long n : {1LL, 3LL, 4LL, 5LL, 31LL, 33LL, 30000LL}) sky<8>(n, places, wrong), sky<2>(n, places, wrong);
    std::printf("sky %lld %lld\n", places, wrong);
    places = wrong = 0;
    for (int warps : {1, 4, 1216, 9728})
        for (long long n : {1LL, 31LL, 1021LL, 9728LL, 9729LL, 700001LL, (1LL << 31) - 320000, (1LL << 31) - 9728,
                            (1LL << 31) - 9727, (1LL << 31) - 1})
            queue(n, warps, places, wrong);
    std::printf("queue %lld %lld\n", places, wrong);
    places = wrong = 0;
    for (long long nn : {1LL, 3LL, 4LL, 5LL, 20479LL, (1LL << 27) - 1, 1LL << 27, (1LL << 27) + 1, 1LL << 28, (1LL << 31) - 1})
        refit(nn, places, wrong);
    std::printf("refit %lld %lld\n", places, wrong);
    return 0;
}
