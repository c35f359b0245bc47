// knn_exact_core.cuh -- device building blocks of the fused exact FP32 k-NN
// kernels (single problem: knn_exact.cu; many problems in one persistent
// launch: knn_batched.cu).  See knn_exact.cu for the algorithm.
#pragma once

#include <atomic>

#include "knn_common.cuh"

namespace knnb200 {

constexpr int EX_BR = 256;       // reference points per tile
constexpr int EX_BD = 16;        // dimensions per pipeline stage
constexpr int EX_CB = 128;       // candidate slots per query (one half tile)
constexpr int EX_WARPS = 16;     // consumer warps
constexpr int EX_QPW = 4;        // queries per warp for k <= 128
constexpr int EX_QPW_K256 = 2;   // queries per warp for 128 < k <= 256
// Four warps of consumers to each scheduler and a warpgroup for the producer, of
// which one thread works.  Each consumer thread takes 112 registers (setmaxnreg):
// launched with 96, 640 x 96 = 61440 >= 128 x 24 + 512 x 112 = 60416.  With 17
// warps of 96 the inner loop and the selection spilled: 10.29 -> 10.07 ms at 131072
// x 4736, d = 256, k = 100; 692 -> 676 us at 16384 x 4096, d = 128, k = 16; 19.3 ->
// 18.8 ms for a batch of 512.
constexpr int EX_THREADS = (EX_WARPS + 4) * 32;
constexpr int EX_LAUNCH_REGS = 96, EX_PRODUCER_REGS = 24, EX_CONSUMER_REGS = 112;
static_assert(128 * EX_PRODUCER_REGS + EX_WARPS * 32 * EX_CONSUMER_REGS <=
                  EX_THREADS * EX_LAUNCH_REGS,
              "the consumers' registers come from the block's own");
// Whether `kern` is launched with the registers that the split counts on (a build
// with fewer would leave its consumers waiting).  Only a good answer is kept: a
// failure to ask, for want of memory to load the kernel say, is this call's alone.
template <auto kern>
bool launch_regs_ok() {
    static std::atomic<bool> known{false};
    if (known.load(std::memory_order_relaxed)) return true;
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, kern) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.numRegs < EX_LAUNCH_REGS) return false;
    known.store(true, std::memory_order_relaxed);
    return true;
}
KNN_DI void producer_regs() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(EX_PRODUCER_REGS));
}
KNN_DI void consumer_regs() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EX_CONSUMER_REGS));
}

template <int QPW, int KCAP>
struct ExCfg {
    static constexpr int BQ = QPW * EX_WARPS;
    // ring depth: what the lists leave of the shared memory
    static constexpr int STAGES = QPW < 4 || KCAP == 32 ? 6 : KCAP == 64 ? 5 : 4;
    static constexpr int Q_FLOATS = EX_BD * BQ;   // query slab of a stage
    static constexpr int R_FLOATS = EX_BD * EX_BR;
    static constexpr int STAGE_FLOATS = Q_FLOATS + R_FLOATS;
    static constexpr int STAGE_BYTES = STAGE_FLOATS * 4;
    // key slots per query: k <= KCAP, one half tile and a margin of 32, so that
    // a selection need not find exactly the k smallest (buf_select)
    static constexpr int REGION = KCAP + EX_CB + 32;
    static constexpr size_t LIST_BYTES = (size_t)BQ * REGION * 8;
    static constexpr size_t TAU_OFFSET = (size_t)STAGES * STAGE_BYTES + LIST_BYTES;
    static constexpr size_t BAR_OFFSET = TAU_OFFSET + BQ * 8;
    static constexpr size_t SMEM = 1024 + BAR_OFFSET + 2 * STAGES * 8 + 16;
    static_assert(STAGE_BYTES % 1024 == 0, "stage alignment");
    static_assert(SMEM <= 232448, "shared memory per CTA");
    static_assert(KCAP % 32 == 0 && (KCAP & (KCAP - 1)) == 0, "KCAP power of two >= 32");
};

KNN_DI void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EX_WARPS * 32) : "memory"); }

// Number of elements of the sorted array L[0..n) (n a power of two) below x.
template <int n>
KNN_DI int rank_pow2(const unsigned long long *L, unsigned long long x) {
    int pos = 0;
#pragma unroll
    for (int step = n / 2; step >= 1; step >>= 1)
        if (L[pos + step - 1] < x) pos += step;
    return pos + (L[pos] < x ? 1 : 0);
}

// Ascending bitonic sort of 32 CPL keys held by one warp, CPL per lane
// (element e = b * 32 + lane in v[b]): lane partners by shuffle, register
// partners in place.
template <int CPL>
KNN_DI void warp_sort(unsigned long long (&v)[CPL], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * CPL; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
                const int rs = stride >> 5;
#pragma unroll
                for (int b = 0; b < CPL; ++b) {
                    if (b & rs) continue;
                    const bool up = (((b << 5) | lane) & size) == 0;
                    const unsigned long long x = v[b], y = v[b | rs];
                    const bool sw = (x > y) == up;
                    v[b] = sw ? y : x;
                    v[b | rs] = sw ? x : y;
                }
            } else {
                const bool lower = (lane & stride) == 0;
#pragma unroll
                for (int b = 0; b < CPL; ++b) {
                    const bool up = (((b << 5) | lane) & size) == 0;
                    const unsigned long long x = v[b];
                    const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, stride);
                    const bool take = (y < x) == (lower == up);
                    v[b] = take ? y : x;
                }
            }
        }
    }
}

// warp_merge for c <= 32 CPL candidates.
template <int KCAP, int CPL>
KNN_DI void warp_merge_n(unsigned long long *L, int c, int k, int lane) {
    constexpr int LPL = KCAP / 32;
    unsigned long long *C = L + KCAP;
    unsigned long long lv[LPL], cv[CPL];
#pragma unroll
    for (int b = 0; b < CPL; ++b) {
        const int t = b * 32 + lane;
        cv[b] = t < c ? C[t] : kKeyInf;
    }
    warp_sort<CPL>(cv, lane);
#pragma unroll
    for (int a = 0; a < LPL; ++a) lv[a] = L[a * 32 + lane];
    __syncwarp();
#pragma unroll
    for (int b = 0; b < CPL; ++b) C[b * 32 + lane] = cv[b];
    __syncwarp();
    int lp[LPL], cp[CPL];
#pragma unroll
    for (int a = 0; a < LPL; ++a) lp[a] = a * 32 + lane + rank_pow2<32 * CPL>(C, lv[a]);
#pragma unroll
    for (int b = 0; b < CPL; ++b) cp[b] = b * 32 + lane + rank_pow2<KCAP>(L, cv[b]);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < LPL; ++a)
        if (lp[a] < k) L[lp[a]] = lv[a];
#pragma unroll
    for (int b = 0; b < CPL; ++b)
        if (b * 32 + lane < c && cp[b] < k) L[cp[b]] = cv[b];
    __syncwarp();
}

// Merge c (<= EX_CB) unsorted candidate keys (L[KCAP .. KCAP+c)) into the
// sorted list L[0..k) held by one warp.  The candidates are sorted in
// registers (32, 64 or 128 of them: a sort of 128 takes 28 exchange steps of
// four keys a lane, one of 32 takes 15 of one) and written back sorted; then
// every key's final position is its index plus its rank in the other sorted
// array (binary search).  Keys are unique (distinct indices), so the positions
// form a permutation; positions >= k are dropped.
template <int KCAP>
KNN_DI void warp_merge(unsigned long long *L, int c, int k, int lane) {
    static_assert(EX_CB == 128, "at most four keys a lane");
    if (c <= 32) warp_merge_n<KCAP, 1>(L, c, k, lane);
    else if (c <= 64) warp_merge_n<KCAP, 2>(L, c, k, lane);
    else warp_merge_n<KCAP, 4>(L, c, k, lane);
}

// ---------------------------------------------------------------------------
// Selection state of one query: an unsorted buffer of REGION key slots and a
// threshold tau; keys >= tau are known not to belong to the k smallest.  A half
// tile's keys below tau are appended; when they would not fit, buf_select finds
// a lower tau and drops what is above it.  Any tau that keeps between k and
// KCAP + 32 keys will do, so it is found by bisection over the distances' bits
// (a count over the buffer for each step, about six steps) instead of sorting:
// about 250 instructions against the 1300 to 1900 of sorting 128 keys and
// merging them into a sorted list of k.  tau lags the keys seen, so more points
// pass, but selections become rare: the gap between them grows geometrically
// as tau tightens.  The buffer is sorted once, at the end of the range.
// ---------------------------------------------------------------------------

// Keep the keys of B[0..c) (c > k + slack) below a tau of which there are at
// least k and at most k + slack, in their order; tau goes to *tau.  Returns
// their number.  One warp; not inlined: its call sites share one copy.
template <int KCAP>
__device__ __noinline__ int buf_select(unsigned long long *B, unsigned long long *tau, int c,
                                       int k, int slack, int lane) {
    constexpr int SL = (KCAP + EX_CB + 32) / 32;
    unsigned long long key[SL];
    uint32_t lo = 0xffffffffu, up = 0;
#pragma unroll
    for (int a = 0; a < SL; ++a) {
        const int t = a * 32 + lane;
        key[a] = t < c ? B[t] : kKeyInf;
        const uint32_t h = (uint32_t)(key[a] >> 32);
        lo = min(lo, h);
        up = max(up, t < c ? h : 0u);
    }
    // invariant: fewer than k keys have a distance below lo, n >= k below up
    lo = __reduce_min_sync(0xffffffffu, lo);
    up = __reduce_max_sync(0xffffffffu, up) + 1u;
    int n = c;
    while (n > k + slack && up - lo > 1u) {
        const uint32_t mid = lo + (up - lo) / 2u;
        int m = 0;
#pragma unroll
        for (int a = 0; a < SL; ++a) m += (uint32_t)(key[a] >> 32) < mid ? 1 : 0;
        m = (int)__reduce_add_sync(0xffffffffu, (unsigned)m);
        if (m >= k) {
            up = mid;
            n = m;
        } else {
            lo = mid;
        }
    }
    unsigned long long cut = (unsigned long long)up << 32;
    if (n > k + slack) {
        // many keys of the one distance lo: bisection over their indices
        // (all different) ends with exactly k at the latest
        unsigned long long a0 = (unsigned long long)lo << 32, a1 = cut;
        while (n > k + slack) {
            const unsigned long long mid = a0 + (a1 - a0) / 2;
            int m = 0;
#pragma unroll
            for (int a = 0; a < SL; ++a) m += key[a] < mid ? 1 : 0;
            m = (int)__reduce_add_sync(0xffffffffu, (unsigned)m);
            if (m >= k) {
                a1 = mid;
                n = m;
            } else {
                a0 = mid;
            }
        }
        cut = a1;
    }
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
    int pos = 0;
#pragma unroll
    for (int a = 0; a < SL; ++a) {
        const bool in = key[a] < cut;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) B[pos + __popc(m & lt)] = key[a];
        pos += __popc(m);
    }
    if (lane == 0) *tau = cut;
    __syncwarp();
    return n;
}

// The k smallest keys of B[0..c), ascending, into B[0..k) (kKeyInf where there
// are fewer).  One warp.
template <int KCAP>
__device__ __noinline__ void buf_finish(unsigned long long *B, unsigned long long *tau, int c,
                                        int k, int lane) {
    constexpr int LPL = KCAP / 32;
    if (c > KCAP) c = buf_select<KCAP>(B, tau, c, k, KCAP - k, lane);
    unsigned long long v[LPL];
#pragma unroll
    for (int a = 0; a < LPL; ++a) v[a] = a * 32 + lane < c ? B[a * 32 + lane] : kKeyInf;
    warp_sort<LPL>(v, lane);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < LPL; ++a) B[a * 32 + lane] = v[a];
    __syncwarp();
}

// Buffer fill of query i (warp-uniform), 16 bits per query.
KNN_DI int nbuf_get(unsigned long long nb, int i) { return (int)((nb >> (16 * i)) & 0xffffu); }
KNN_DI unsigned long long nbuf_set(unsigned long long nb, int i, int v) {
    return (nb & ~(0xffffull << (16 * i))) | ((unsigned long long)v << (16 * i));
}

// Start of a reference range: empty buffers; queries beyond the set have a
// threshold that nothing passes.
template <int QPW>
KNN_DI void select_start(unsigned long long *wt, unsigned long long &nb, int q0, int Q, int lane) {
    nb = 0;
    if (lane < QPW) wt[lane] = q0 + lane < Q ? kKeyInf : 0ull;
    __syncwarp();
}

// End of a reference range: every query's buffer sorted.  (Not unrolled.)
template <int QPW, int KCAP>
KNN_DI void select_finish(unsigned long long *wl, unsigned long long *wt, unsigned long long nb,
                          int k, int lane) {
    static_assert(QPW <= 4, "buffer fills packed in one word");
    constexpr int REGION = ExCfg<QPW, KCAP>::REGION;
#pragma unroll 1
    for (int i = 0; i < QPW; ++i)
        buf_finish<KCAP>(wl + i * REGION, wt + i, nbuf_get(nb, i), k, lane);
}

// How many keys more than k a selection may leave: up to KCAP + 32 - k fit beside
// the next half tile's survivors.  Few make a lower threshold, which later tiles
// pass less often, for a step or two more of the bisection: with k / 8 + 3, 18783
// -> 18540 us for a batch of 512 problems (k to 64), 560 -> 536 at 100000 x 4736, d = 5
// and 894 -> 863 at d = 20 (k = 20), 926 -> 914 at 65536 x 2048, d = 64, k = 200, 609 ->
// 610.6 at 16384 x 4096, d = 128, k = 16; k / 4 + 4 to k / 3 + 3 give two thirds of that.
// Lists of 128 keys (100 of them wanted) leave 60 as they did: 9854 us at 131072 x
// 4736, d = 256, against 9964.
template <int KCAP>
KNN_DI int select_slack(int k) {
    return KCAP == 128 ? KCAP + 32 - k : min(KCAP + 32 - k, k / 8 + 3);
}

// Filter one half tile (4 reference points per lane) against the thresholds of
// the queries in hitq and append the survivors to their buffers.  A query
// whose buffer was selected here is tested again with its new threshold: of a
// list's first half tiles, all of whose points pass, later ones then add few.
// nb packs the warp-uniform buffer fills.  d2(i, j) gives the squared
// distance of query i to the lane's j-th point.  With LB, only keys >= lb[i]
// are selected: pass p of a k > 256 problem keeps the 256 smallest keys above
// the ones earlier passes returned.
template <int QPW, int KCAP, bool LB, typename D2>
KNN_DI void select_half_lb(unsigned long long *wl, unsigned long long *wt,
                           unsigned long long &nb, D2 d2, uint32_t rbase, int N, int k, int lane,
                           uint32_t hitq, const unsigned long long (&lb)[QPW]) {
    constexpr int REGION = ExCfg<QPW, KCAP>::REGION;
    auto passing = [&](int i) {
        const unsigned long long tau = wt[i];
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t idx = rbase + j;
            const unsigned long long key = make_key(d2(i, j), idx);
            bool p = (idx < (uint32_t)N) && key < tau;
            if (LB) p = p && key >= lb[i];
            m |= (p ? 1u : 0u) << j;
        }
        return m;
    };
    uint32_t pm[QPW];
    uint32_t full_mask = 0;   // queries whose buffer cannot take the survivors
#pragma unroll
    for (int i = 0; i < QPW; ++i) {
        pm[i] = 0;
        if (!((hitq >> i) & 1u)) continue;
        pm[i] = passing(i);
        const int m_i = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(pm[i]));
        if (nbuf_get(nb, i) + m_i > REGION) full_mask |= 1u << i;
    }
    if (full_mask) {
        __syncwarp();
#pragma unroll 1
        for (int i = 0; i < QPW; ++i)
            if ((full_mask >> i) & 1u)
                nb = nbuf_set(nb, i, buf_select<KCAP>(wl + i * REGION, wt + i, nbuf_get(nb, i), k,
                                                      select_slack<KCAP>(k), lane));
#pragma unroll
        for (int i = 0; i < QPW; ++i)
            if ((full_mask >> i) & 1u) pm[i] = passing(i);
    }
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < QPW; ++i) {
        if (__ballot_sync(0xffffffffu, pm[i] != 0) == 0) continue;
        unsigned long long *cb = wl + i * REGION;
        int c = nbuf_get(nb, i);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool p = (pm[i] >> j) & 1u;
            const unsigned m = __ballot_sync(0xffffffffu, p);
            if (p) cb[c + __popc(m & lt)] = make_key(d2(i, j), rbase + j);
            c += __popc(m);
        }
        nb = nbuf_set(nb, i, c);
    }
    __syncwarp();
}

// The warp's QPW queries of one dimension (one broadcast load).
template <int QPW>
KNN_DI void load_queries(float (&q)[QPW], const float *src) {
    static_assert(QPW == 4 || QPW == 2 || QPW == 1, "one load");
    if constexpr (QPW == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(src);
        q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;
    } else if constexpr (QPW == 2) {
        const float2 v = *reinterpret_cast<const float2 *>(src);
        q[0] = v.x; q[1] = v.y;
    } else {
        q[0] = *src;
    }
}

// One dimension of the lane's QPW x 8 block.
template <int QPW>
KNN_DI void consume_dim(f32x2_t (&acc)[QPW][4], const float *rs, const float *qs) {
    // 16-byte loads straight into packed pairs (x, y), (z, w)
    const ulonglong2 ra = *reinterpret_cast<const ulonglong2 *>(rs);
    const ulonglong2 rb = *reinterpret_cast<const ulonglong2 *>(rs + 128);
    const f32x2_t r0 = ra.x, r1 = ra.y, r2 = rb.x, r3 = rb.y;
    float q[QPW];
    load_queries<QPW>(q, qs);
#pragma unroll
    for (int i = 0; i < QPW; ++i) {
        const f32x2_t qq = f2_pack(q[i], q[i]);
        f32x2_t t;
        t = f2_sub(r0, qq); acc[i][0] = f2_fma(t, t, acc[i][0]);
        t = f2_sub(r1, qq); acc[i][1] = f2_fma(t, t, acc[i][1]);
        t = f2_sub(r2, qq); acc[i][2] = f2_fma(t, t, acc[i][2]);
        t = f2_sub(r3, qq); acc[i][3] = f2_fma(t, t, acc[i][3]);
    }
}

// Groups of four dimensions in the last stage of d dimensions.
__host__ __device__ inline int last_stage_groups(int d) { return ((d - 1) % EX_BD) / 4 + 1; }

// Consume the n_dchunks pipeline stages of one reference tile: the lane's
// QPW x 8 block of squared distances accumulates sum_d (r_d - q_d)^2 with a
// rounded sub and a fused multiply-add per dimension, in increasing d (the
// order of the reference's compute_distances loop, code/knncuda.cu:77-80).
// Bound by the FP32 pipe: 32 packed operations a warp and dimension take 16
// cycles of an SM.  The shared loads return 128 B a cycle whatever lanes share:
// two loads of references and one of the four queries take 12.  (Queries kept
// as (q, q) pairs in shared memory saved the register moves but took 16: 298
// against 289 ms at 2^20 x 16384, d = 256, k = 100, 814 against 764 us at
// 16384 x 4096, d = 128, k = 16.)
// PARTIAL: the last stage takes only `tail` groups of four dimensions
// (last_stage_groups); 1143 -> 884 us at 100000 x 4736, d = 20, k = 20, 712 -> 548 at
// d = 5, 1074 -> 982 at 30000 x 4736, d = 100.
// `it` is the running stage counter of the CTA's ring.  Returns false (warp-
// uniformly) if a wait timed out or another warp aborted.
template <int QPW, int KCAP, bool PARTIAL>
KNN_DI bool consume_ref_tile(f32x2_t (&acc)[QPW][4], const float *stages, uint64_t *full,
                             uint64_t *empty, volatile int *abort_flag, int &it, int n_dchunks,
                             int tail, int warp, int lane, int *status) {
    using C = ExCfg<QPW, KCAP>;
#pragma unroll
    for (int i = 0; i < QPW; ++i)
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[i][p] = 0ull;
    for (int dc = 0; dc < n_dchunks; ++dc, ++it) {
        const int s = it % C::STAGES;
        const bool got = mbar_wait(&full[s], (it / C::STAGES) & 1);
        // warp-uniform decision: every lane leaves together or none does.
        // No per-stage check of the abort flag: when another warp gives up,
        // the producer stops refilling and this wait ends by its time limit.
        if (__any_sync(0xffffffffu, !got)) {
            if (lane == 0) {
                atomicMax(status, (int)kDevTimeoutFull);
                *abort_flag = 1;
            }
            return false;
        }
        const float *qs = stages + (size_t)s * C::STAGE_FLOATS + warp * QPW;
        const float *rs = stages + (size_t)s * C::STAGE_FLOATS + C::Q_FLOATS + lane * 4;
        if (!PARTIAL || dc + 1 < n_dchunks || tail == EX_BD / 4) {
#pragma unroll
            for (int dd = 0; dd < EX_BD; ++dd)
                consume_dim<QPW>(acc, rs + dd * EX_BR, qs + dd * C::BQ);
        } else {
            // the last chunk's dimensions, in fours: the zeros beyond them would
            // add exact zeros
#pragma unroll 1
            for (int g = 0; g < tail; ++g) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    consume_dim<QPW>(acc, rs + (4 * g + e) * EX_BR, qs + (4 * g + e) * C::BQ);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
    }
    return true;
}

// Select both halves of a consumed tile (reference points rt*256 + ...).
// Most tiles hold no candidate of most queries, so each lane first compares
// the smallest of its 8 distances (as bits: the order of the keys, whatever
// the index) with the threshold's: about one instruction per pair instead of
// six for the key comparisons of every pair.
template <int QPW, int KCAP, bool LB>
KNN_DI void select_tile(unsigned long long *wl, unsigned long long *wt, unsigned long long &nb,
                        f32x2_t (&acc)[QPW][4], int rt, int N, int k, int lane,
                        const unsigned long long (&lb)[QPW]) {
    auto d2 = [&](int i, int j) {
        return (j & 1) ? f2_hi(acc[i][j >> 1]) : f2_lo(acc[i][j >> 1]);
    };
    uint32_t hitq = 0;
#pragma unroll
    for (int i = 0; i < QPW; ++i) {
        uint32_t b[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) b[j] = __float_as_uint(d2(i, j));
        const uint32_t m = min(min(min(min(b[0], b[1]), b[2]), min(min(b[3], b[4]), b[5])),
                               min(b[6], b[7]));
        const uint32_t tau = (uint32_t)(wt[i] >> 32);
        hitq |= __any_sync(0xffffffffu, m <= tau) ? 1u << i : 0u;
    }
    if (!hitq) return;
    const uint32_t rb0 = (uint32_t)rt * EX_BR + lane * 4;
    select_half_lb<QPW, KCAP, LB>(wl, wt, nb, d2, rb0, N, k, lane, hitq, lb);
    select_half_lb<QPW, KCAP, LB>(
        wl, wt, nb, [&](int i, int j) { return d2(i, 4 + j); }, rb0 + 128, N, k, lane, hitq, lb);
}

// ---------------------------------------------------------------------------
// Merge of the per-split sorted key lists of one query, by one warp: a running
// list of the k smallest keys takes one split's list after the other.  Only the
// keys below the running k-th key (a prefix, since the list is sorted; about
// k / t keys of the t-th list) are merged: every key's position is its index
// plus its rank in the other list.  The next list's keys are loaded while this
// one is merged.
// ---------------------------------------------------------------------------
template <int KCAP, int NC>   // the first n <= 32 NC keys of v
KNN_DI void merge_prefix(unsigned long long *L, unsigned long long *C,
                         const unsigned long long (&v)[KCAP / 32], int n, int k, int lane) {
    constexpr int LPL = KCAP / 32;
    unsigned long long lv[LPL];
    int lp[LPL], cp[NC];
#pragma unroll
    for (int b = 0; b < NC; ++b) C[b * 32 + lane] = b * 32 + lane < n ? v[b] : kKeyInf;
#pragma unroll
    for (int a = 0; a < LPL; ++a) lv[a] = L[a * 32 + lane];
    __syncwarp();
    // equal keys (entries without a point) keep the running list's first
#pragma unroll
    for (int a = 0; a < LPL; ++a) lp[a] = a * 32 + lane + rank_pow2<32 * NC>(C, lv[a]);
#pragma unroll
    for (int b = 0; b < NC; ++b) cp[b] = b * 32 + lane + rank_pow2<KCAP>(L, v[b] + 1);
    __syncwarp();
#pragma unroll
    for (int a = 0; a < LPL; ++a)
        if (lp[a] < k) L[lp[a]] = lv[a];
#pragma unroll
    for (int b = 0; b < NC; ++b)
        if (b * 32 + lane < n && cp[b] < k) L[cp[b]] = v[b];
    __syncwarp();
}

// L (KCAP keys) receives the k smallest keys of the lists t0, t0 + step, ...
// below S; list t starts at src + t * pitch.  C: KCAP keys of scratch.
template <int KCAP>
KNN_DI void merge_lists(unsigned long long *L, unsigned long long *C,
                        const unsigned long long *src, size_t pitch, int t0, int step, int S,
                        int k, int lane) {
    constexpr int LPL = KCAP / 32;
    unsigned long long nxt[LPL], cur[LPL];
    auto load = [&](unsigned long long (&v)[LPL], int t) {
#pragma unroll
        for (int a = 0; a < LPL; ++a) {
            const int j = a * 32 + lane;
            v[a] = t < S && j < k ? src[(size_t)t * pitch + j] : kKeyInf;
        }
    };
    load(cur, t0);
#pragma unroll
    for (int a = 0; a < LPL; ++a) L[a * 32 + lane] = cur[a];
    __syncwarp();
    load(nxt, t0 + step);
    for (int t = t0 + step; t < S; t += step) {
#pragma unroll
        for (int a = 0; a < LPL; ++a) cur[a] = nxt[a];
        load(nxt, t + step);
        const unsigned long long tau = L[k - 1];
        int n = 0;
#pragma unroll
        for (int a = 0; a < LPL; ++a)
            n += __popc(__ballot_sync(0xffffffffu, cur[a] < tau));
        if (n == 0) continue;
        if (LPL == 1 || n <= 32) merge_prefix<KCAP, 1>(L, C, cur, n, k, lane);
        else merge_prefix<KCAP, LPL>(L, C, cur, n, k, lane);
    }
}

}  // namespace knnb200
