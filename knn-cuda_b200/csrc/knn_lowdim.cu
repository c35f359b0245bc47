// knn_lowdim.cu -- exact FP32 brute-force k-NN for low dimension (d <= 4) and
// small k (k <= 16), e.g. 3-D point clouds.
//
// At d = 3 the distance of a pair costs three subtractions and three fused
// multiply-adds, so the work is dominated by issue, not by data: the tiled
// kernel's 16-dimension stages would waste 13/16 of its arithmetic.  Here a
// warp holds QPW queries; its lanes take four reference points each, 128
// consecutive ones a step (one 16-byte load per dimension and lane), as packed
// pairs for sub.f32x2 / fma.f32x2.  A step's distances are first compared with
// the query's k-th smallest so far (three minima, one compare and one vote for
// four points); survivors enter the query's sorted list, which lies across the
// lanes (knn_lane_list.cuh).
//
// Arithmetic: acc = fma(t0, t0, 0), acc = fma(t_i, t_i, acc) for i = 1..d-1,
// t_i = r_i - q_i -- the fused exact kernel's chain (its zero-padded
// dimensions add exact zeros), so distances are bit-identical to it.
// Selection keeps the smallest (distance, index) keys: equal distances keep
// the lower index first -- the reference's rule (code/knncuda.cu:172, :178).
//
// Bound by the FP32 pipe: 24 lane operations per four points at d = 3.  One
// thread per query with register lists, the layout before this one, took 29.1
// ms at 2^20 x 65536, d = 3, k = 8, where this one takes 22.2, and left most of
// the GPU idle at smaller sizes (d = 3, k = 8): 267 -> 32 us at 1000 x 4000, 527 -> 55
// at 65536 x 400, 2179 -> 134 at 2^20 x 100, 1566 -> 851 at 2^18 x 8192.
//
// Many queries against few points run one thread a pair of queries
// (knn_lowdim_thread_kernel): a warp's list costs it the same few thousand cycles
// a query however few the points are.
//
// Large clouds are searched in space (knn_space.cu) where the caller has the
// scratch for it; this kernel then answers the few queries that search leaves
// over.
#include <algorithm>
#include <cmath>

#include "../../include/knn_b200.h"
#include "knn_exact_core.cuh"
#include "knn_kernels.h"
#include "knn_lane_list.cuh"

namespace knnb200 {

constexpr int LD_WARPS = 8;      // warps per block
constexpr int LD_STEP = 128;     // reference points per step of a warp
constexpr int LD_MAX_K = 16;

// A block takes LD_WARPS / WPQ groups of QPW queries and one split of the
// reference set; with WPQ = LD_WARPS its warps share the split of one group
// and merge their lists.
template <int D, int QPW, int WPQ>
__global__ void __launch_bounds__(32 * LD_WARPS)
    knn_lowdim_kernel(const float *__restrict__ ref, int N, long long ldr,
                      const float *__restrict__ qry, int Q, long long ldq, int k, int n_splits,
                      float *__restrict__ out_dist, int *__restrict__ out_idx, long long ld_out,
                      unsigned long long *__restrict__ part, QuerySubset subset) {
    constexpr int GROUPS = LD_WARPS / WPQ, QPB = GROUPS * QPW;
    __shared__ unsigned long long lists[LD_WARPS][QPW][32], merged[GROUPS][QPW][32];
    __shared__ unsigned long long keys[LD_WARPS][LD_STEP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int group = warp / WPQ;
    // with a subset: its queries, and the blocks loop over the (query block,
    // split) pairs; otherwise one pair per block
    const int nq = subset.count ? *subset.count : Q;
    if (subset.count) n_splits = subset.splits(nq, n_splits);
    const long long n_items = ((long long)nq + QPB - 1) / QPB * n_splits;
    const long long steps = ((long long)N + LD_STEP - 1) / LD_STEP;
    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int split = (int)(item % n_splits);
        // (unsigned: the last block's queries may lie beyond the largest int)
        const unsigned q0 = (unsigned)(item / n_splits) * QPB + group * QPW;
        // this warp's steps
        const long long parts = (long long)n_splits * WPQ;
        const long long mypart = (long long)split * WPQ + warp % WPQ;
        const long long s0 = steps * mypart / parts, s1 = steps * (mypart + 1) / parts;
        float q[QPW][D];
        unsigned long long mine[QPW], tau[QPW];
#pragma unroll
        for (int i = 0; i < QPW; ++i) {
            const unsigned qi = q0 + i;
            const int col = qi < (unsigned)nq ? (subset.list ? subset.list[qi] : (int)qi) : -1;
#pragma unroll
            for (int dd = 0; dd < D; ++dd) q[i][dd] = col >= 0 ? qry[(size_t)dd * ldq + col] : 0.f;
            mine[i] = kKeyNone;
            tau[i] = col >= 0 ? kKeyNone : 0ull;   // nothing passes a query beyond the set
        }
        auto load = [&](float4 (&r)[D], long long s) {
            const long long p = s * LD_STEP + lane * 4;
#pragma unroll
            for (int dd = 0; dd < D; ++dd) {
                const float *src = ref + (size_t)dd * ldr + p;
                if (p + 3 < N) {
                    r[dd] = *reinterpret_cast<const float4 *>(src);
                } else {
                    // the set's last points (NaN: never selected)
                    const float none = __int_as_float(0x7fc00000);
                    r[dd].x = p < N ? src[0] : none;
                    r[dd].y = p + 1 < N ? src[1] : none;
                    r[dd].z = p + 2 < N ? src[2] : none;
                    r[dd].w = none;
                }
            }
        };
        float4 nxt[D];
        if (s0 < s1) load(nxt, s0);
        for (long long s = s0; s < s1; ++s) {
            f32x2_t ra[D], rb[D];
#pragma unroll
            for (int dd = 0; dd < D; ++dd) {
                ra[dd] = f2_pack(nxt[dd].x, nxt[dd].y);
                rb[dd] = f2_pack(nxt[dd].z, nxt[dd].w);
            }
            if (s + 1 < s1) load(nxt, s + 1);
#pragma unroll
            for (int i = 0; i < QPW; ++i) {
                f32x2_t a, b;
#pragma unroll
                for (int dd = 0; dd < D; ++dd) {
                    const f32x2_t qq = f2_pack(q[i][dd], q[i][dd]);
                    const f32x2_t ta = f2_sub(ra[dd], qq), tb = f2_sub(rb[dd], qq);
                    a = f2_fma(ta, ta, dd ? a : 0ull);
                    b = f2_fma(tb, tb, dd ? b : 0ull);
                }
                const float d4[4] = {f2_lo(a), f2_hi(a), f2_lo(b), f2_hi(b)};
                const float m = fminf(fminf(d4[0], d4[1]), fminf(d4[2], d4[3]));
                // (strictly: a step's indices are above all earlier ones)
                if (!__any_sync(0xffffffffu, m < key_dist2(tau[i]))) continue;
                lane_list_add4(mine[i], tau[i], d4, m, (uint32_t)(s * LD_STEP + lane * 4), k,
                               lane, keys[warp]);
            }
        }
        if (WPQ > 1) {
#pragma unroll
            for (int i = 0; i < QPW; ++i) lists[warp][i][lane] = mine[i];
            __syncthreads();
            if (warp % WPQ == 0) {
#pragma unroll 1
                for (int i = 0; i < QPW; ++i) {
                    merge_lists<32>(merged[group][i], lists[warp][i], &lists[warp][i][0],
                                    (size_t)QPW * 32, 0, 1, WPQ, k, lane);
                }
            }
            __syncwarp();
        }
        // results: sqrt into the k x Q layout, or this split's sorted keys for
        // the split merge
        if (warp % WPQ == 0) {
#pragma unroll
            for (int i = 0; i < QPW; ++i) {
                const unsigned qi = q0 + i;
                if (qi >= (unsigned)nq || lane >= k) continue;
                const unsigned long long key = WPQ > 1 ? merged[group][i][lane] : mine[i];
                if (n_splits == 1) {
                    const int col = subset.list ? subset.list[qi] : (int)qi;
                    out_dist[(size_t)lane * ld_out + col] = sqrtf(key_dist2(key));
                    out_idx[(size_t)lane * ld_out + col] = key_index(key);
                } else {
                    part[((size_t)split * Q + qi) * k + lane] = key;
                }
            }
        }
        if (WPQ > 1) __syncthreads();   // the lists are rewritten
    }
}

// Every thread holds two queries (packed for sub.f32x2 / fma.f32x2) and their sorted
// lists of K in registers; the block streams the reference points through a
// double-buffered tile of shared memory, each coordinate stored twice, (r, r), so
// that a 64-bit load is a packed operand, and every thread scans the tile in the
// order of the indices: a point enters a list if it is strictly nearer than the
// last entry and passes only strictly farther ones, so equal distances keep the
// lower index first.  Bound by issue: the insertions of a warp's 64 lists diverge,
// about 100 of the 150 instructions a point costs a warp at 128 points (K = 8).
// One warp a query took 880 us for 3 10^6 queries against 16 points (d = 1, k = 1),
// this kernel 127; 1043 and 299 for 10^6 against 128 (d = 3, k = 8), 3166 and 883
// for 3 10^6 against 64 (d = 4, k = 16).  (Four queries a thread: 0 to 30 % slower.)
constexpr int LT_THREADS = 256;
constexpr int LT_TILE = 512;   // reference points per shared tile
template <int D, int K>
__global__ void __launch_bounds__(LT_THREADS, 2)
    knn_lowdim_thread_kernel(const float *__restrict__ ref, int N, long long ldr,
                             const float *__restrict__ qry, int Q, long long ldq, int k,
                             float *__restrict__ out_dist, int *__restrict__ out_idx,
                             long long ld_out) {
    __shared__ float2 tile[2][D][LT_TILE];
    const int tid = threadIdx.x;
    // (unsigned: the last block's may lie beyond the largest int)
    const unsigned qid[2] = {blockIdx.x * 2 * LT_THREADS + tid,
                             blockIdx.x * 2 * LT_THREADS + LT_THREADS + tid};
    const unsigned nq = (unsigned)Q;
    f32x2_t q[D];
#pragma unroll
    for (int dd = 0; dd < D; ++dd)
        q[dd] = f2_pack(qid[0] < nq ? qry[(size_t)dd * ldq + qid[0]] : 0.f,
                        qid[1] < nq ? qry[(size_t)dd * ldq + qid[1]] : 0.f);
    float ld[2][K];
    int li[2][K];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < K; ++j) {
            ld[m][j] = INFINITY;
            li[m][j] = -1;
        }
    constexpr int PER = LT_TILE / LT_THREADS;   // points per thread per tile load
    float pre[D][PER];
    auto fetch = [&](int t) {
#pragma unroll
        for (int dd = 0; dd < D; ++dd)
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const long long r = (long long)t * LT_TILE + u * LT_THREADS + tid;
                pre[dd][u] = r < N ? ref[(size_t)dd * ldr + r] : 0.f;
            }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int dd = 0; dd < D; ++dd)
#pragma unroll
            for (int u = 0; u < PER; ++u)
                tile[buf][dd][u * LT_THREADS + tid] = make_float2(pre[dd][u], pre[dd][u]);
    };
    const int tiles = (int)(((long long)N + LT_TILE - 1) / LT_TILE);
    fetch(0);
    stash(0);
    __syncthreads();
    for (int t = 0; t < tiles; ++t) {
        if (t + 1 < tiles) fetch(t + 1);
        const int rbase = t * LT_TILE, valid = min(LT_TILE, N - rbase);
        for (int j = 0; j < valid; ++j) {
            f32x2_t acc;
#pragma unroll
            for (int dd = 0; dd < D; ++dd) {
                const f32x2_t x = f2_sub(*reinterpret_cast<const f32x2_t *>(&tile[t & 1][dd][j]),
                                         q[dd]);
                acc = f2_fma(x, x, dd ? acc : 0ull);
            }
            const float d2[2] = {f2_lo(acc), f2_hi(acc)};
            if (!(d2[0] < ld[0][K - 1] || d2[1] < ld[1][K - 1])) continue;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                if (!(d2[m] < ld[m][K - 1])) continue;
#pragma unroll
                for (int i = K - 1; i > 0; --i) {
                    const bool past = d2[m] < ld[m][i - 1], here = d2[m] < ld[m][i];
                    ld[m][i] = past ? ld[m][i - 1] : here ? d2[m] : ld[m][i];
                    li[m][i] = past ? li[m][i - 1] : here ? rbase + j : li[m][i];
                }
                if (d2[m] < ld[m][0]) {
                    ld[m][0] = d2[m];
                    li[m][0] = rbase + j;
                }
            }
        }
        if (t + 1 < tiles) stash((t + 1) & 1);
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (qid[m] >= nq) continue;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            if (j >= k) break;
            out_dist[(size_t)j * ld_out + qid[m]] = sqrtf(ld[m][j]);
            out_idx[(size_t)j * ld_out + qid[m]] = li[m][j];
        }
    }
}

namespace {

// Splits that callers' scratch is sized for, and the kernel's own choice.
struct LowdimShape {
    int max_splits;
    bool thread;   // knn_lowdim_thread_kernel
    int qpw, wpq, splits;
};

// Whether one thread a pair of queries takes less than warps, in us.  A thread's
// points cost 0.22 (lists of 8; 16: 0.37) each while the blocks are one an SM, then
// in proportion to the queries, less for more points, of which fewer enter a list.
// A warp's query costs about as much up to 128 points, then more slowly than in
// proportion.  Fitted to 1236 problems of 16 to 16000 points, 1000 to 3 10^6 queries
// and k = 1 to 16; thread / warp measured at d = 3, k = 8: 24 / 50 with 16 x 50000,
// 34 / 48 with 64 x 50000, 48 / 46 with 128 x 50000, 145 / 223 with 128 x 400000, 108 /
// 80 with 512 x 50000, 831 / 1143 with 512 x 10^6.
bool thread_pays(int N, int Q, int k) {
    if (N > 1024) return false;
    const double few = 128.0 / std::max(N, 128);
    const double point = k <= 8 ? std::max(0.22, 0.12 + 2.0e-6 * Q * std::pow(few, 0.2))
                                : std::max(0.37, 0.2 + 4.4e-6 * Q * std::pow(few, 0.12));
    const double query = (0.25e-3 + 0.035e-3 * k) * std::pow(few, -0.55);
    return N * point < Q * query;
}

bool lowdim_shape(int N, int Q, int d, int k, int num_sms, LowdimShape &s) {
    if (d < 1 || d > 4 || k < 1 || k > LD_MAX_K) return false;
    const int bq = 256 * (k <= 8 ? 4 : 2);
    const int n_rtiles = (N + 511) / 512;
    const int qtiles = (Q + bq - 1) / bq;
    // two blocks of bq queries per SM; splits fill whole waves, each >= 8 tiles
    const int slots = 2 * num_sms;
    int best = 1;
    double best_t = 1e300;
    const int max_s = std::max(1, std::min({256, n_rtiles / 8, (160 * 1024) / (8 * k)}));
    for (int S = 1; S <= max_s; ++S) {
        const long long ctas = (long long)qtiles * S;
        const double t = (double)((ctas + slots - 1) / slots) * ((double)n_rtiles / S + 0.5);
        if (t < best_t * 0.999) {
            best_t = t;
            best = S;
        }
    }
    s.max_splits = best;
    // Few queries take a whole block each.  More queries to a warp share its loads,
    // but the code that adds to their lists no longer fits the instruction cache
    // with four: that pays only where few points enter a list, in large problems (at
    // d = 3, k = 8, two / four queries a warp: 1074 / 1153 us at 8000 x 200000, 185 /
    // 216 at 16384 x 14000, 506 / 488 at 65536 x 14000, 1768 / 1477 at 262144 x 14000;
    // one: 2418 there, 45 / 46 with two at 4000 x 4000).
    const int want = num_sms * 48;   // warps that keep the GPU busy
    s.wpq = 1;
    if (Q < 300 || (Q < 1200 && N < 131072)) {
        s.qpw = 1;
        if (N >= (Q <= 512 ? 256 : 1000)) s.wpq = LD_WARPS;
    } else if (N < 32768) {
        s.qpw = Q < 5000 ? 1 : 2;
    } else {
        s.qpw = (double)N * Q >= 1e9 ? 4 : 2;
    }
    // splits of 8192 points and more: each starts its lists anew
    const long long warps = ((long long)Q + s.qpw - 1) / s.qpw * s.wpq;
    const long long fill = s.wpq > 1 ? want / 2 / warps : (want + warps - 1) / warps;
    s.splits = (int)std::max<long long>(
        1, std::min({(long long)s.max_splits, fill, (long long)N / 8192}));
    s.thread = thread_pays(N, Q, k);
    return true;
}

template <int D>
cudaError_t launch_ld(const ExactProblem &p, const LowdimShape &s, unsigned long long *part,
                      const QuerySubset &subset, cudaStream_t st) {
    auto go = [&](auto kern, int qpb) {
        const long long items = ((long long)p.Q + qpb - 1) / qpb * s.splits;
        // a subset is usually small or empty: blocks that loop
        const long long grid = subset.count ? std::min<long long>(items, 4 * p.num_sms) : items;
        kern<<<(unsigned)grid, 32 * LD_WARPS, 0, st>>>(p.ref, p.N, p.ldr, p.qry, p.Q, p.ldq, p.k,
                                                       s.splits, p.out_dist, p.out_idx, p.ld_out,
                                                       part, subset);
        return cudaGetLastError();
    };
    if (s.thread) {
        const unsigned blocks = (unsigned)(((long long)p.Q + 2 * LT_THREADS - 1) /
                                           (2 * LT_THREADS));
        const auto kern = p.k <= 8 ? knn_lowdim_thread_kernel<D, 8>
                                   : knn_lowdim_thread_kernel<D, LD_MAX_K>;
        kern<<<blocks, LT_THREADS, 0, st>>>(p.ref, p.N, p.ldr, p.qry, p.Q, p.ldq, p.k, p.out_dist,
                                            p.out_idx, p.ld_out);
        return cudaGetLastError();
    }
    if (s.wpq > 1) return go(knn_lowdim_kernel<D, 1, LD_WARPS>, 1);
    if (s.qpw == 4) return go(knn_lowdim_kernel<D, 4, 1>, 4 * LD_WARPS);
    if (s.qpw == 2) return go(knn_lowdim_kernel<D, 2, 1>, 2 * LD_WARPS);
    return go(knn_lowdim_kernel<D, 1, 1>, LD_WARPS);
}

}  // namespace

bool lowdim_applies(int N, int Q, int d, int k) {
    LowdimShape s;
    return lowdim_shape(N, Q, d, k, 148, s);
}

size_t lowdim_scratch_bytes(int N, int Q, int d, int k, int num_sms) {
    LowdimShape s;
    if (!lowdim_shape(N, Q, d, k, num_sms, s)) return 0;
    return s.max_splits > 1 ? (size_t)s.max_splits * Q * k * 8 : 0;
}

int lowdim_plan_splits(int N, int Q, int d, int k, int num_sms) {
    LowdimShape s;
    return lowdim_shape(N, Q, d, k, num_sms, s) ? s.max_splits : 0;
}

int lowdim_plan_route(int N, int Q, int d, int k, int num_sms) {
    LowdimShape s;
    if (!lowdim_shape(N, Q, d, k, num_sms, s)) return -1;
    return space_applies(N, Q, d, k) ? KNNB200_ROUTE_CLOUD_SPACE
           : s.thread                ? KNNB200_ROUTE_CLOUD_THREAD
                                     : KNNB200_ROUTE_CLOUD_WARP;
}

int launch_lowdim(const ExactProblem &p, cudaStream_t st) {
    LowdimShape s;
    if (!lowdim_shape(p.N, p.Q, p.d, p.k, p.num_sms, s)) return kErrUnsupported;
    if (p.force_splits > 0) s.splits = std::min(p.force_splits, std::min((p.N + 511) / 512, 256));
    // a large cloud is searched in space; the brute force then answers the
    // queries that search left over
    QuerySubset sub;
    if (p.space && space_applies(p.N, p.Q, p.d, p.k)) {
        const int rc = launch_space(p, st, &sub);
        if (rc != kOk) return rc;
        s.thread = false;
        s.qpw = 4;
        s.wpq = 1;
        s.splits = s.max_splits;
        sub.slots = 2 * p.num_sms;
        sub.steps = (p.N + LD_STEP - 1) / LD_STEP;
    }
    if (s.thread) s.splits = 1;
    // as many splits as the scratch holds lists of (it may have been sized for the
    // larger first chunk of a call, whose plan has fewer)
    s.splits = (int)std::min<size_t>(
        s.splits, std::max<size_t>(1, p.scratch_bytes / ((size_t)p.Q * p.k * 8)));
    unsigned long long *part = static_cast<unsigned long long *>(p.scratch);
    cudaError_t e;
    switch (p.d) {
        case 1: e = launch_ld<1>(p, s, part, sub, st); break;
        case 2: e = launch_ld<2>(p, s, part, sub, st); break;
        case 3: e = launch_ld<3>(p, s, part, sub, st); break;
        default: e = launch_ld<4>(p, s, part, sub, st); break;
    }
    if (e != cudaSuccess) return kErrLaunch;
    if (p.timer) p.timer->mark(st, kPhaseExactMain);
    if (s.splits > 1) {
        const int rc = launch_split_merge(part, s.splits, p.Q, p.k, p.out_dist, p.out_idx,
                                          p.ld_out, st, 0, nullptr, sub);
        if (rc != kOk) return rc;
        if (p.timer) p.timer->mark(st, kPhaseExactMerge);
    }
    return kOk;
}

}  // namespace knnb200
