// knn_exact.cu -- fused exact FP32 k-NN (direct form) for sm_100a.
//
// Replaces the reference chain compute_distances (code/knncuda.cu:20-91) ->
// modified_insertion_sort (:143-189) -> compute_sqrt (:200-205) with ONE
// kernel: the ref_nb x query_nb distance matrix never reaches HBM.
//
//   * A CTA owns BQ queries (one query tile) and one contiguous slice
//     ("split") of the reference set.  Reference tiles of 256 points x 16
//     dimensions and the matching 16 x BQ query slab are brought into shared
//     memory by TMA (one producer warp, an mbarrier ring of 4 to 6 stages).
//   * 16 consumer warps; warp w owns QPW queries, lane l owns the 8
//     reference points {4l..4l+3, 128+4l..128+4l+3} of each tile, so every
//     lane accumulates a QPW x 8 block of squared distances in registers as
//     sum_d (r_d - q_d)^2 with one rounding per sub and one fused
//     multiply-add per dimension, in increasing d -- the arithmetic and
//     order of the reference's compute_distances inner loop
//     (code/knncuda.cu:77-80), so squared distances are bit-identical to it.
//   * Selection is warp-local.  Each query has an unsorted buffer of candidate
//     keys (distance, index) and a threshold in shared memory.  After each tile
//     the warp ballots the keys below the threshold into the buffer; when they
//     would not fit, a bisection over the buffered distances lowers the
//     threshold to one that keeps the k smallest and few more (buf_select).
//     The buffer is sorted once, at the end of the CTA's range.
//     Ordering by the 64-bit key (distance bits, index) reproduces the
//     reference's tie rule: equal distances keep the lower index
//     (code/knncuda.cu:172, :178).
//   * Where that grid's waves do not come out even, the tiles of all query tiles
//     are laid end to end and cut into one range a CTA instead (TileRanges).
//   * With one split the kernel writes sqrt(distance) and the index straight
//     into the k x query_nb output; with several splits it writes each
//     split's sorted keys to scratch and knn_merge_splits_kernel merges them.
//   * k > 256 (the reference's insertion sort has no limit on k,
//     code/knncuda.cu:143-189) runs in passes over the whole set: pass p
//     keeps the 256 smallest keys at or above a per-query lower bound (one
//     more than the last key of pass p - 1) and writes output rows
//     256 p .. 256 p + 255.  Keys are unique, so the passes together return
//     exactly the k smallest keys in order, with the same distances and tie
//     order as a single pass.
#include <algorithm>
#include <cstdio>
#include <type_traits>

#include "../../include/knn_b200.h"
#include "knn_exact_core.cuh"
#include "knn_kernels.h"

namespace knnb200 {

// RANGES: the CTA takes the whole tiles [u0, u1) of all query tiles' reference
// tiles laid end to end (TileRanges), which may cross from one query tile into
// the next; the ring runs on across the border.
template <int QPW, int KCAP, bool LB, bool PARTIAL, bool RANGES>
__global__ void __launch_bounds__(EX_THREADS, 1)
    knn_exact_kernel(const __grid_constant__ CUtensorMap tm_ref,
                     const __grid_constant__ CUtensorMap tm_qry, ExactArgs a) {
    using C = ExCfg<QPW, KCAP>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float *stages = reinterpret_cast<float *>(base);
    unsigned long long *lists =
        reinterpret_cast<unsigned long long *>(base + (size_t)C::STAGES * C::STAGE_BYTES);
    uint64_t *full = reinterpret_cast<uint64_t *>(base + C::BAR_OFFSET);
    uint64_t *empty = full + C::STAGES;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(empty + C::STAGES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qtile = blockIdx.x, split = blockIdx.y;
    const int t0 = (int)((long long)a.n_rtiles * split / a.n_splits);
    const int t1 = (int)((long long)a.n_rtiles * (split + 1) / a.n_splits);
    const long long u0 = RANGES ? a.ranges.begin(blockIdx.x) : 0;
    const long long u1 = RANGES ? a.ranges.begin(blockIdx.x + 1) : 0;
    const int total = (RANGES ? (int)(u1 - u0) : t1 - t0) * a.n_dchunks;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], EX_WARPS);
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    __syncthreads();

    if (warp >= EX_WARPS) {
        producer_regs();
        if (warp > EX_WARPS) return;
        // ---------------- producer warp: one thread issues all TMA loads ----
        if (lane == 0) {
            prefetch_tensormap(&tm_ref);
            prefetch_tensormap(&tm_qry);
            int issued = 0;
            for (int it = 0; it < total; ++it) {
                const int s = it % C::STAGES;
                if (it >= C::STAGES && !mbar_wait(&empty[s], ((it / C::STAGES) - 1) & 1)) {
                    atomicMax(a.status, (int)kDevTimeoutEmpty);
                    *abort_flag = 1;
                    break;
                }
                if (*abort_flag) break;
                float *qs = stages + (size_t)s * C::STAGE_FLOATS;
                float *rs = qs + C::Q_FLOATS;
                int rt = t0 + it / a.n_dchunks, qt = qtile;
                const int dc = it % a.n_dchunks;
                if (RANGES) {
                    const long long u = u0 + it / a.n_dchunks;
                    qt = (int)(u / a.n_rtiles);
                    rt = (int)(u % a.n_rtiles);
                }
                mbar_arrive_expect_tx(&full[s], C::STAGE_BYTES);
                tma_load_2d(qs, &tm_qry, &full[s], qt * C::BQ, dc * EX_BD);
                tma_load_2d(rs, &tm_ref, &full[s], rt * EX_BR, dc * EX_BD);
                issued = it + 1;
            }
            // Never leave with copies in flight: wait for the last issued stages.
            for (int it = max(0, issued - C::STAGES); it < issued; ++it)
                if (!mbar_wait(&full[it % C::STAGES], (it / C::STAGES) & 1))
                    atomicMax(a.status, (int)kDevTimeoutDrain);
        }
        return;
    }

    // -------------------- consumer warps ------------------------------------
    consumer_regs();
    unsigned long long *wl = lists + (size_t)warp * QPW * C::REGION;
    unsigned long long *wt =
        reinterpret_cast<unsigned long long *>(base + C::TAU_OFFSET) + warp * QPW;
    unsigned long long nb;   // buffer fills
    if constexpr (RANGES) {
        const unsigned long long no_lb[QPW] = {};
        const int tail = last_stage_groups(a.d);
        int it = 0;
        for (long long u = u0; u < u1;) {
            const int qt = (int)(u / a.n_rtiles), r0 = (int)(u % a.n_rtiles);
            const int r1 = (int)min((long long)a.n_rtiles, r0 + (u1 - u));
            const int qw = qt * C::BQ + warp * QPW;
            select_start<QPW>(wt, nb, qw, a.Q, lane);
            for (int rt = r0; rt < r1; ++rt) {
                f32x2_t acc[QPW][4];
                if (!consume_ref_tile<QPW, KCAP, PARTIAL>(acc, stages, full, empty, abort_flag,
                                                          it, a.n_dchunks, tail, warp, lane,
                                                          a.status))
                    return;
                select_tile<QPW, KCAP, false>(wl, wt, nb, acc, rt, a.N, a.k, lane, no_lb);
            }
            select_finish<QPW, KCAP>(wl, wt, nb, a.k, lane);
            const int slot = (int)blockIdx.x - a.ranges.owner((long long)qt * a.n_rtiles);
            for (int i = 0; i < QPW; ++i) {
                if (qw + i >= a.Q) break;
                unsigned long long *dst = a.part + ((size_t)slot * a.Q + qw + i) * a.k;
                for (int j = lane; j < a.k; j += 32) dst[j] = wl[i * C::REGION + j];
            }
            __syncwarp();   // the buffers are rewritten
            u += r1 - r0;
        }
        return;
    }
    select_start<QPW>(wt, nb, qtile * C::BQ + warp * QPW, a.Q, lane);
    unsigned long long lbk[QPW];
#pragma unroll
    for (int i = 0; i < QPW; ++i) {
        const int q = qtile * C::BQ + warp * QPW + i;
        lbk[i] = (LB && q < a.Q) ? a.lb[q] : 0ull;
    }

    int it = 0;
    const int tail = last_stage_groups(a.d);
    for (int rt = t0; rt < t1; ++rt) {
        f32x2_t acc[QPW][4];
        if (!consume_ref_tile<QPW, KCAP, PARTIAL>(acc, stages, full, empty, abort_flag, it, a.n_dchunks,
                                         tail, warp, lane, a.status))
            break;
        select_tile<QPW, KCAP, LB>(wl, wt, nb, acc, rt, a.N, a.k, lane, lbk);
    }
    select_finish<QPW, KCAP>(wl, wt, nb, a.k, lane);

    consumer_sync();
    if (*abort_flag) return;

    const int q0 = qtile * C::BQ;
    if (a.n_splits == 1) {
        // Epilogue: sqrt and the reference's k x query_nb layout, coalesced
        // along queries.
        for (int e = threadIdx.x; e < a.k * C::BQ; e += EX_WARPS * 32) {
            const int j = e / C::BQ, qi = e - j * C::BQ, q = q0 + qi;
            if (q < a.Q) {
                const unsigned long long key = lists[(size_t)qi * C::REGION + j];
                a.out_dist[(size_t)(a.row0 + j) * a.ld_out + q] = sqrtf(key_dist2(key));
                a.out_idx[(size_t)(a.row0 + j) * a.ld_out + q] = key_index(key);
                if (a.lb_out && j == a.k - 1) a.lb_out[q] = key + 1;
            }
        }
    } else {
        for (int i = 0; i < QPW; ++i) {
            const int q = q0 + warp * QPW + i;
            if (q >= a.Q) break;
            unsigned long long *dst = a.part + ((size_t)split * a.Q + q) * a.k;
            for (int j = lane; j < a.k; j += 32) dst[j] = wl[i * C::REGION + j];
        }
    }
}

// Copy of a query set whose rows TMA cannot read in place (base or row pitch
// not a multiple of 16 bytes).
__global__ void copy_queries_kernel(const float *__restrict__ src, int Q, long long lds,
                                    float *__restrict__ dst, long long ldd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int dd = blockIdx.y;
    if (i < Q) dst[(size_t)dd * ldd + i] = src[(size_t)dd * lds + i];
}

// Merge the per-split sorted key lists of each query (merge_lists).  A block of
// eight warps takes 8 / WPQ consecutive queries, WPQ warps each: one warp a
// query, or all eight on one (each merges every eighth list, then the first
// one merges the eight results) where the queries alone do not fill the GPU
// and the lists are many.
constexpr int MG_WARPS = 8;
template <int KCAP, int WPQ>
__global__ void __launch_bounds__(32 * MG_WARPS)
    knn_merge_splits_kernel(const unsigned long long *__restrict__ part, int S, int Q, int k,
                            float *__restrict__ out_dist, int *__restrict__ out_idx,
                            long long ld_out, int row0, unsigned long long *__restrict__ lb_out,
                            QuerySubset subset, TileRanges ranges) {
    constexpr int QPB = MG_WARPS / WPQ;
    __shared__ unsigned long long lists[MG_WARPS][KCAP], scratch[MG_WARPS][KCAP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nq = subset.count ? *subset.count : Q;
    if (subset.count) S = subset.splits(nq, S);
    if (subset.count && S == 1) return;   // written without lists
    for (int q0 = blockIdx.x * QPB; q0 < nq; q0 += gridDim.x * QPB) {
        const int q = q0 + warp / WPQ;
        if (q < nq) {
            merge_lists<KCAP>(lists[warp], scratch[warp], part + (size_t)q * k, (size_t)Q * k,
                              warp % WPQ, WPQ, ranges.ctas ? ranges.lists(q) : S, k, lane);
        }
        __syncthreads();
        if (WPQ > 1) {
            if (warp == 0)
                merge_lists<KCAP>(scratch[0], scratch[1], lists[0], KCAP, 0, 1, WPQ, k, lane);
            __syncthreads();
        }
        // rows of the k x query_nb output, QPB queries wide
        for (int e = threadIdx.x; e < k * QPB; e += 32 * MG_WARPS) {
            const int j = e / QPB, qi = q0 + e % QPB;
            if (qi >= nq) continue;
            const unsigned long long key = WPQ > 1 ? scratch[0][j] : lists[e % QPB][j];
            const int col = subset.list ? subset.list[qi] : qi;
            out_dist[(size_t)(row0 + j) * ld_out + col] = sqrtf(key_dist2(key));
            out_idx[(size_t)(row0 + j) * ld_out + col] = key_index(key);
            if (lb_out && j == k - 1) lb_out[col] = key + 1;
        }
        __syncthreads();   // the lists are rewritten
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

struct ExactShape {
    int qpw, kcap, bq, splits, n_rtiles, n_dchunks;
    TileRanges ranges;      // ctas = 0: the grid of qtiles x splits
    int range_lists = 0;    // lists a query of the ranges has, at most
    size_t smem;
};

template <int QPW, int KCAP>
void shape_of(ExactShape &s) {
    using C = ExCfg<QPW, KCAP>;
    s.qpw = QPW;
    s.kcap = KCAP;
    s.bq = C::BQ;
    s.smem = C::SMEM;
}

template <int QPW>
void shape_for_k(int k, ExactShape &s) {
    if (k <= 32) shape_of<QPW, 32>(s);
    else if (k <= 64) shape_of<QPW, 64>(s);
    else shape_of<QPW, 128>(s);
}

// Ranks selected by one pass of the kernel: k <= 256 in one pass, larger k
// in passes of 256 (the last one may be shorter).
constexpr int kPassRanks = 256;

bool choose_shape(int N, int Q, int d, int k_all, int num_sms, ExactShape &s) {
    if (k_all < 1) return false;
    const int k = std::min(k_all, kPassRanks);
    // up to 32 queries: tiles of 32 or 16, two or one to a warp, which cut the
    // arithmetic on padding and the selections a warp makes one after the other:
    // with tiles of 64, 14.8 us at 1000 x 16 (d = 32, k = 10), now 7.3; 531 at 10^6
    // x 1 (d = 128, k = 10), now 278; 266 at 200000 x 20 (d = 256, k = 100), now 164
    if (k > 128) shape_of<EX_QPW_K256, 256>(s);
    else if (Q <= 16) shape_for_k<1>(k, s);
    else if (Q <= 32) shape_for_k<2>(k, s);
    else shape_for_k<EX_QPW>(k, s);
    s.n_rtiles = (N + EX_BR - 1) / EX_BR;
    s.n_dchunks = (d + EX_BD - 1) / EX_BD;
    const int qtiles = (Q + s.bq - 1) / s.bq;
    // Split the reference set so that the grid fills whole waves of one CTA
    // per SM.  Modelled time: waves x (tiles per split + fixed selection
    // warm-up cost of about 256/d tiles per split).
    const double warm = 256.0 / (s.n_dchunks * EX_BD);
    int best = 1;
    double best_t = 1e300;
    // up to 256 splits and 20480 list entries per query
    int max_s = std::min(s.n_rtiles, std::min(256, (160 * 1024) / (8 * k)));
    // keep the per-split partial lists under 1 GiB of scratch
    const long long per_split = (long long)Q * k * 8;
    max_s = (int)std::max<long long>(1, std::min<long long>(max_s, (1ll << 30) / per_split));
    for (int S = 1; S <= max_s; ++S) {
        const long long ctas = (long long)qtiles * S;
        const long long waves = (ctas + num_sms - 1) / num_sms;
        const double t = (double)waves * ((double)s.n_rtiles / S + warm);
        if (t < best_t * 0.999) {
            best_t = t;
            best = S;
        }
    }
    s.splits = best;
    // The grid leaves SMs idle where its waves do not come out even.  One range
    // of tiles a CTA (TileRanges) gives every SM the same work, but most CTAs
    // then hold parts of two query tiles and warm up twice.  Modelled time as
    // above, in whole tiles; taken where it is less by 3 %.  Measured over 84
    // shapes of d = 8 to 512 and k = 5 to 100: at a modelled ratio below 0.97 the
    // ranges take 0.78 to 0.975 of the grid's time (675 -> 609 us at 16384 x 4096, d
    // = 128, k = 16: 128 CTAs of the grid; 1771 -> 1635 at 17149 x 2865, d = 512),
    // from 0.97 to 1 they take 0.94 to 1.03, above 1 up to 1.2.
    s.ranges = TileRanges();
    const long long units = (long long)qtiles * s.n_rtiles;
    if (s.qpw != EX_QPW || k_all > 128 || units < num_sms) return true;
    const long long per = (units + num_sms - 1) / num_sms;
    const long long parts = (per + s.n_rtiles - 2) / s.n_rtiles + 1;   // query tiles of a CTA
    const long long waves = ((long long)qtiles * best + num_sms - 1) / num_sms;
    const double t_grid = (double)waves * ((s.n_rtiles + best - 1) / best + warm);
    const long long lists = (s.n_rtiles - 1) / (units / num_sms) + 2;   // at most, of a query
    if (per + parts * warm < 0.97 * t_grid && lists <= max_s &&
        per * s.n_dchunks < (1ll << 31)) {
        s.ranges.ctas = num_sms;
        s.ranges.bq = s.bq;
        s.ranges.n_rtiles = s.n_rtiles;
        s.ranges.units = units;
        s.range_lists = (int)lists;
    }
    return true;
}

template <int QPW, int KCAP, bool LB, bool PARTIAL, bool RANGES>
cudaError_t launch_v(const CUtensorMap &mr, const CUtensorMap &mq, const ExactArgs &a,
                     int qtiles, cudaStream_t st) {
    using C = ExCfg<QPW, KCAP>;
    constexpr auto kern = knn_exact_kernel<QPW, KCAP, LB, PARTIAL, RANGES>;
    if (!launch_regs_ok<kern>()) return cudaErrorLaunchOutOfResources;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)C::SMEM);
    if (e != cudaSuccess) return e;
    const dim3 grid = RANGES ? dim3(a.ranges.ctas) : dim3(qtiles, a.n_splits);
    kern<<<grid, EX_THREADS, C::SMEM, st>>>(mr, mq, a);
    return cudaGetLastError();
}

template <int QPW, int KCAP, bool LB = false>
cudaError_t launch_t(const CUtensorMap &mr, const CUtensorMap &mq, const ExactArgs &a,
                     int qtiles, cudaStream_t st) {
    // Whole stages run either variant.  The one with the test for a short stage
    // measured faster with lists of 128 keys and four stages or more a tile (277.3
    // -> 272.2 ms at 2^20 x 16384, d = 256, k = 100; 1440 -> 1434 us at 65536 x 4736, d
    // = 64) and slower below (867 -> 883 at d = 32; 793 -> 809 with k = 32): the
    // compiler schedules the stage differently around the branch.
    const bool partial = last_stage_groups(a.d) < EX_BD / 4 ||
                         (KCAP == 128 && QPW == EX_QPW && a.n_dchunks >= 4);
    if constexpr (QPW == EX_QPW && !LB && KCAP <= 128) {
        if (a.ranges.ctas)
            return partial ? launch_v<QPW, KCAP, LB, true, true>(mr, mq, a, qtiles, st)
                           : launch_v<QPW, KCAP, LB, false, true>(mr, mq, a, qtiles, st);
    }
    return partial ? launch_v<QPW, KCAP, LB, true, false>(mr, mq, a, qtiles, st)
                   : launch_v<QPW, KCAP, LB, false, false>(mr, mq, a, qtiles, st);
}

template <int QPW>
cudaError_t launch_k(int kcap, const CUtensorMap &mr, const CUtensorMap &mq, const ExactArgs &a,
                     int qtiles, cudaStream_t st) {
    switch (kcap) {
        case 32: return launch_t<QPW, 32>(mr, mq, a, qtiles, st);
        case 64: return launch_t<QPW, 64>(mr, mq, a, qtiles, st);
        default: return launch_t<QPW, 128>(mr, mq, a, qtiles, st);
    }
}

}  // namespace

// Row pitch of the query copy, in floats.
static long long qcopy_pitch(int Q) { return ((long long)Q + 31) / 32 * 32; }

int launch_split_merge(const unsigned long long *part, int S, int Q, int k, float *out_dist,
                       int *out_idx, long long ld_out, cudaStream_t st, int row0,
                       unsigned long long *lb_out, const QuerySubset &subset,
                       const TileRanges &ranges) {
    if (k > kPassRanks) return kErrUnsupported;
    // all eight warps on one query: 14.6 us against 51.9 with one warp a query at
    // 40 queries and 148 lists of 50 keys, 15.4 against 22.7 at 300 queries and 29
    // lists of 100; at 1000 queries and 9 lists one warp a query takes 10.7
    const bool wide = Q <= 1024 && S >= 16;
    auto go = [&](auto kern, int qpb) {
        // a subset is usually empty: few blocks, which loop if it is not
        const int all = (Q + qpb - 1) / qpb, blocks = subset.count ? std::min(all, 592) : all;
        kern<<<blocks, 32 * MG_WARPS, 0, st>>>(part, S, Q, k, out_dist, out_idx, ld_out, row0,
                                               lb_out, subset, ranges);
        return cudaGetLastError() == cudaSuccess ? (int)kOk : (int)kErrLaunch;
    };
    auto pick = [&](auto cap) {
        constexpr int C = decltype(cap)::value;
        return wide ? go(knn_merge_splits_kernel<C, MG_WARPS>, 1)
                    : go(knn_merge_splits_kernel<C, 1>, MG_WARPS);
    };
    if (k <= 32) return pick(std::integral_constant<int, 32>());
    if (k <= 64) return pick(std::integral_constant<int, 64>());
    if (k <= 128) return pick(std::integral_constant<int, 128>());
    return pick(std::integral_constant<int, 256>());
}

// Scratch of the exact path: room for two copies of the queries (one is used,
// and only when theirs cannot be read in place; the size is what callers of
// the allocation-free entry plan with), 256 bytes of alignment, the per-split
// key lists of one pass when the reference set is split, and for k > 256 the
// per-query lower-bound keys of the passes.
static size_t exact_need(const ExactShape &s, int Q, int d, int k) {
    const int kp = std::min(k, kPassRanks);
    const size_t dup = (size_t)d * qcopy_pitch(Q) * 2 * sizeof(float);
    const size_t part = s.splits > 1 ? (size_t)s.splits * Q * kp * 8 : 0;
    const size_t lb = k > kPassRanks ? (size_t)Q * 8 : 0;
    return dup + 256 + part + lb;
}

// Where a call's lists lie in its scratch: after the copy of the queries, if
// there is one.
static size_t lists_offset(int Q, int d, bool copied) {
    return copied ? ((size_t)d * qcopy_pitch(Q) * sizeof(float) + 255) & ~size_t(255) : 0;
}

size_t exact_scratch_bytes(int N, int Q, int d, int k, int num_sms) {
    if (lowdim_applies(N, Q, d, k)) return lowdim_scratch_bytes(N, Q, d, k, num_sms);
    ExactShape s;
    if (!choose_shape(N, Q, d, k, num_sms, s)) return 0;
    return exact_need(s, Q, d, k);
}

// Scratch of the ranges: their lists, after the copy of the queries.  The room of
// the copies holds them in most cases.
static size_t ranges_need(const ExactShape &s, int Q, int d, int k, bool copied) {
    return lists_offset(Q, d, copied) + (size_t)s.range_lists * Q * k * 8;
}

size_t exact_scratch_wanted(int N, int Q, int d, int k, int num_sms) {
    const size_t need = exact_scratch_bytes(N, Q, d, k, num_sms);
    ExactShape s;
    if (lowdim_applies(N, Q, d, k) || !choose_shape(N, Q, d, k, num_sms, s) || !s.ranges.ctas)
        return need;
    const size_t want = ranges_need(s, Q, d, k, true);
    return want > need + (size_t(64) << 20) ? need : std::max(need, want);
}

bool exact_supported_k(int k) { return k >= 1; }

int launch_exact(const ExactProblem &p, cudaStream_t st) {
    if (lowdim_applies(p.N, p.Q, p.d, p.k)) return launch_lowdim(p, st);
    ExactShape s;
    if (!choose_shape(p.N, p.Q, p.d, p.k, p.num_sms, s)) return kErrUnsupported;
    if (p.force_splits > 0) s.splits = std::min(p.force_splits, std::min(s.n_rtiles, 256));
    const bool copied = (reinterpret_cast<uintptr_t>(p.qry) & 15) || p.ldq % 4;
    const size_t part_off = lists_offset(p.Q, p.d, copied);
    const size_t lb_bytes = p.k > kPassRanks ? (size_t)p.Q * 8 : 0;
    if (part_off + lb_bytes > p.scratch_bytes) return kErrScratch;
    // not where the split is given, or the scratch has no room for the lists
    if (s.ranges.ctas &&
        (p.force_splits > 0 || ranges_need(s, p.Q, p.d, p.k, copied) > p.scratch_bytes))
        s.ranges = TileRanges();
    if (s.ranges.ctas) {
        s.splits = s.range_lists;
    } else {
        // as many splits as the scratch holds lists of: it may have been sized for
        // more queries than these (the last chunk of a call, the queries that the
        // tensor path leaves over), whose plan has fewer
        const size_t per_split = (size_t)p.Q * std::min(p.k, kPassRanks) * 8;
        const size_t fit = (p.scratch_bytes - part_off - lb_bytes) / per_split;
        s.splits = (int)std::min<size_t>(s.splits, std::max<size_t>(1, fit));
    }
    const size_t lb_off = part_off + (s.splits > 1 ? (size_t)s.splits * p.Q *
                                                         std::min(p.k, kPassRanks) * 8
                                                   : 0);
    unsigned char *sb = static_cast<unsigned char *>(p.scratch);
    unsigned long long *part = reinterpret_cast<unsigned long long *>(sb + part_off);
    unsigned long long *lb = reinterpret_cast<unsigned long long *>(sb + lb_off);
    const float *qry = p.qry;
    long long ldq = p.ldq;
    if (copied) {
        float *copy = static_cast<float *>(p.scratch);
        ldq = qcopy_pitch(p.Q);
        // rows on gridDim.y (at most 65535 of them a launch)
        for (int d0 = 0; d0 < p.d; d0 += 65535) {
            const dim3 grid((p.Q + 255) / 256, std::min(65535, p.d - d0));
            copy_queries_kernel<<<grid, 256, 0, st>>>(p.qry + (size_t)d0 * p.ldq, p.Q, p.ldq,
                                                      copy + (size_t)d0 * ldq, ldq);
        }
        if (cudaGetLastError() != cudaSuccess) return kErrLaunch;
        qry = copy;
    }

    CUtensorMap mr, mq;
    if (!encode_f32_2d(&mr, p.ref, (uint64_t)p.N, (uint64_t)p.d, (uint64_t)p.ldr, EX_BR, EX_BD) ||
        !encode_f32_2d(&mq, qry, (uint64_t)p.Q, (uint64_t)p.d, (uint64_t)ldq, s.bq, EX_BD))
        return kErrTensorMap;

    ExactArgs a;
    a.N = p.N;
    a.Q = p.Q;
    a.d = p.d;
    a.n_rtiles = s.n_rtiles;
    a.n_splits = s.splits;
    a.ranges = s.ranges;
    a.n_dchunks = s.n_dchunks;
    a.out_dist = p.out_dist;
    a.out_idx = p.out_idx;
    a.ld_out = p.ld_out;
    a.part = part;
    a.status = p.status;
    a.lb = lb;
    const int qtiles = (p.Q + s.bq - 1) / s.bq;
    const bool multi = p.k > kPassRanks;
    // ranks [row0, row0 + a.k) per pass
    for (int row0 = 0; row0 < p.k; row0 += kPassRanks) {
        a.k = std::min(kPassRanks, p.k - row0);
        a.row0 = row0;
        a.lb_out = (multi && row0 + a.k < p.k) ? lb : nullptr;
        cudaError_t e;
        if (multi) {
            // pass 0 has no lower bound; every later pass starts above the
            // last key of the one before
            e = row0 == 0 ? launch_t<EX_QPW_K256, 256, false>(mr, mq, a, qtiles, st)
                          : launch_t<EX_QPW_K256, 256, true>(mr, mq, a, qtiles, st);
        } else {
            if (s.kcap == 256) e = launch_t<EX_QPW_K256, 256>(mr, mq, a, qtiles, st);
            else if (s.qpw == 1) e = launch_k<1>(s.kcap, mr, mq, a, qtiles, st);
            else if (s.qpw == 2) e = launch_k<2>(s.kcap, mr, mq, a, qtiles, st);
            else e = launch_k<EX_QPW>(s.kcap, mr, mq, a, qtiles, st);
        }
        if (e != cudaSuccess) return kErrLaunch;
        if (p.timer) p.timer->mark(st, kPhaseExactMain);
        if (s.splits > 1) {
            const int rc = launch_split_merge(a.part, s.splits, p.Q, a.k, p.out_dist, p.out_idx,
                                              p.ld_out, st, row0, a.lb_out, QuerySubset(),
                                              s.ranges);
            if (rc != kOk) return rc;
            if (p.timer) p.timer->mark(st, kPhaseExactMerge);
        }
    }
    return kOk;
}

int exact_plan_splits(int N, int Q, int d, int k, int num_sms) {
    if (lowdim_applies(N, Q, d, k)) return lowdim_plan_splits(N, Q, d, k, num_sms);
    ExactShape s;
    return choose_shape(N, Q, d, k, num_sms, s) ? s.splits : 0;
}

int exact_plan_route(int N, int Q, int d, int k, int num_sms) {
    if (lowdim_applies(N, Q, d, k)) return lowdim_plan_route(N, Q, d, k, num_sms);
    ExactShape s;
    if (!choose_shape(N, Q, d, k, num_sms, s)) return -1;
    return s.ranges.ctas ? KNNB200_ROUTE_RANGES : KNNB200_ROUTE_GRID;
}

}  // namespace knnb200
