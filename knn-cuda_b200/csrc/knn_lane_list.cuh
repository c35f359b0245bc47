// knn_lane_list.cuh -- the k <= 32 smallest keys of one query, one per lane of
// a warp: lane j holds the j-th smallest key, tau is the k-th.
#pragma once

#include "knn_common.cuh"

namespace knnb200 {

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
    // (a key that an earlier one pushed out ends up behind the k-th)
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        const unsigned long long x = __shfl_sync(0xffffffffu, key, src);
        const int pos = __popc(__ballot_sync(0xffffffffu, mine < x));
        const unsigned long long up = __shfl_up_sync(0xffffffffu, mine, 1);
        mine = lane < pos ? mine : lane == pos ? x : up;
    }
    tau = __shfl_sync(0xffffffffu, mine, k - 1);
}

// The k-th smallest of the lanes' values (non-negative, no NaN).
KNN_DI float lane_kth(float x, int k, int lane) {
    uint32_t v = __float_as_uint(x);
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, v, stride);
            v = ((lane & stride) == 0) == ((lane & size) == 0) ? min(v, o) : max(v, o);
        }
    return __uint_as_float(__shfl_sync(0xffffffffu, v, k - 1));
}

// Add the four points idx .. idx + 3 of each lane, at the distances d with the
// minimum m; all indices are above those in the list.  Where many pass -- a list's
// first points, or points that come ever nearer -- only those up to the k-th
// smallest of the lanes' minima can matter: they are gathered through buf (128 keys
// of the warp's own) and added together, with one sort of 32-bit values and one of
// keys instead of four of keys: 8294 -> 2952 us for 20000 queries against 65536
// points in the order of their one coordinate, 154 -> 108 for 50000 queries against
// 1000 random ones at d = 3, k = 8.
KNN_DI void lane_list_add4(unsigned long long &mine, unsigned long long &tau, const float (&d)[4],
                           float m, uint32_t idx, int k, int lane, unsigned long long *buf) {
    const float td = key_dist2(tau);
    const int hits = __popc(__ballot_sync(0xffffffffu, m < td));
    if (hits == 0) return;
    if (hits <= 8) {
#pragma unroll
        for (int j = 0; j < 4; ++j) lane_list_add(mine, tau, finite_key(d[j], idx + j), k, lane);
        return;
    }
    const float lim = hits >= k ? lane_kth(m < td ? m : td, k, lane) : td;
    const unsigned lt = (1u << lane) - 1u;
    int c = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const bool in = d[j] < td && d[j] <= lim;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) buf[c + __popc(b & lt)] = make_key(d[j], idx + j);
        c += __popc(b);
    }
    __syncwarp();
    for (int t = 0; t < c; t += 32)
        lane_list_add(mine, tau, t + lane < c ? buf[t + lane] : kKeyInf, k, lane);
    __syncwarp();
}

}  // namespace knnb200
