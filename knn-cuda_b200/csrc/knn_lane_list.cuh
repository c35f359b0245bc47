// knn_lane_list.cuh -- the k <= 32 smallest keys of one query, one per lane of
// a warp: lane j holds the j-th smallest key, tau is the k-th.
#pragma once

#include "knn_common.cuh"

namespace knnb200 {

constexpr int LL_MAX_K = 32;
// An entry without a point: distance +inf, index -1.
constexpr unsigned long long kKeyNone = (0x7f800000ull << 32) | 0xffffffffull;

// Key of a point; points at an infinite or NaN distance are no neighbours.
KNN_DI unsigned long long finite_key(float d2, uint32_t idx) {
    return d2 < INFINITY ? make_key(d2, idx) : kKeyInf;
}

// Add each lane's key (kKeyInf: none; keys are unique).
KNN_DI void lane_list_add(unsigned long long &mine, unsigned long long &tau,
                          unsigned long long key, int k, int lane) {
    unsigned m = __ballot_sync(0xffffffffu, key < tau);
    if (m == 0) return;
    if (__popc(m) > 8) {
        // many at once: sort them and merge the two sorted lists (the 32
        // smallest of both are the smaller of each pair list[j], new[31 - j],
        // a bitonic sequence)
        if (key >= tau) key = kKeyInf;
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, stride);
                const bool up = (lane & size) == 0, lower = (lane & stride) == 0;
                key = ((o < key) == (lower == up)) ? o : key;
            }
        key = __shfl_xor_sync(0xffffffffu, key, 31);
        mine = key < mine ? key : mine;
#pragma unroll
        for (int stride = 16; stride > 0; stride >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, mine, stride);
            mine = ((o < mine) == ((lane & stride) == 0)) ? o : mine;
        }
        tau = __shfl_sync(0xffffffffu, mine, k - 1);
        return;
    }
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const unsigned long long x = __shfl_sync(0xffffffffu, key, src);
        if (x >= tau) continue;
        const int pos = __popc(__ballot_sync(0xffffffffu, mine < x));
        const unsigned long long up = __shfl_up_sync(0xffffffffu, mine, 1);
        mine = lane < pos ? mine : lane == pos ? x : up;
        tau = __shfl_sync(0xffffffffu, mine, k - 1);
    }
}

}  // namespace knnb200
