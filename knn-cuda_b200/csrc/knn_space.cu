// knn_space.cu -- exact FP32 k-NN for point clouds (d <= 4, k <= 16) that are
// large enough to be put in spatial order first.
//
// In a few dimensions nearly all pairs of a brute force are far from each
// other.  Here the reference points are sorted into a grid along a space-
// filling order, 32 consecutive points form a leaf with its bounding box,
// 32 leaves a node and 32 nodes a top entry.  One warp searches one query: it
// starts with the leaf at the query's own place, which gives a threshold, and
// then visits, nearest box first, the boxes that are not farther than the k-th
// distance found so far.
//
// The results are those of the brute-force kernels, bit for bit.  Distances
// use the same chain, acc = fma(t_i, t_i, acc) with t_i = r_i - q_i.  A box's
// lower bound runs the same chain on the distances to its faces; rounding is
// monotone, so the bound is not above the rounded distance of any point in
// the box, with no margin needed.  Keys (distance bits, index) are unique, so
// the k smallest of them do not depend on the order of the visits; a box at
// exactly the k-th distance is entered when it holds a smaller index.  Points
// at an infinite or NaN distance are never neighbours (their entries stay
// +inf, -1), as in the low-dimension kernel.
//
// The grid only orders the points, so its rounding does not matter.  Where the
// order separates them badly a query gives up after `cap` leaves, or at once
// where a quarter of the points share a cell (a few outliers that stretch the
// grid), and joins a list that the brute-force kernel answers, on the device,
// with no read-back.  Such a query pays for both: points on a sphere and queries near
// its centre take 0.32 to 0.96 of the brute force that ran before the search, all
// queries exactly at the centre up to 1.06 (2^20 points, 4096 queries).
//
// At 2^20 points, d = 3, 65536 queries and k = 8 a call takes 314 us against 22.9
// ms for the brute force: 76 us to order the points (counting and scattering 24
// each, their cell counters' atomics), 214 us to search, bound by its chain of
// box tests and short lists (about 1500 instructions a query) with 48 warps an SM
// to hide the loads.
#include <algorithm>

#include "knn_common.cuh"
#include "knn_kernels.h"
#include "knn_lane_list.cuh"

namespace knnb200 {

namespace {

constexpr int SP_MAX_BITS = 20;      // at most 2^20 grid cells
constexpr int SP_SCAN = 4096;        // counters per block of the scan
constexpr int SP_WARPS = 8;          // queries per block of the search

// Order-preserving bits of a float, and back.
KNN_DI uint32_t sp_ord(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
KNN_DI float sp_unord(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// The grid: extent of the finite coordinates of each dimension, cut in half
// bit by bit, always along the dimension whose cells are longest, so that the
// cells are near cubes whatever the shape of the cloud.  The bits in that
// order, most significant first, are a cell's number.
struct SpaceGrid {
    float lo[4], scale[4];
    int bits[4];
    unsigned long long order;   // 2 bits per step: its dimension, step 0 lowest
    int steps;
};

template <int D>
KNN_DI void sp_grid(SpaceGrid &out, const volatile uint32_t *bbox, int steps) {
    SpaceGrid g;
    double len[4];
#pragma unroll
    for (int d = 0; d < 4; ++d) g.lo[d] = g.scale[d] = 0.f, g.bits[d] = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const uint32_t a = ~bbox[d], b = bbox[4 + d];   // ~0 / 0: no finite coordinate
        const float lo = a <= b ? sp_unord(a) : 0.f, hi = a <= b ? sp_unord(b) : 0.f;
        g.lo[d] = lo;
        len[d] = (double)hi - (double)lo;
        g.scale[d] = (float)len[d];
    }
    g.order = 0;
    g.steps = steps;
    for (int s = 0; s < steps; ++s) {
        int best = 0;
        double bl = -1.0;
#pragma unroll
        for (int d = 0; d < D; ++d)
            if (len[d] > bl) {
                bl = len[d];
                best = d;
            }
#pragma unroll
        for (int d = 0; d < D; ++d)
            if (d == best) {
                len[d] *= 0.5;
                ++g.bits[d];
            }
        g.order |= (unsigned long long)best << (2 * s);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const float cells = (float)(1 << g.bits[d]);
        g.scale[d] = g.scale[d] > 0.f ? cells / g.scale[d] : 0.f;
    }
    out = g;
}

template <int D>
KNN_DI uint32_t sp_cell(const SpaceGrid &g, const float (&x)[D]) {
    uint32_t c[4] = {0, 0, 0, 0};
    int left[4] = {0, 0, 0, 0};
#pragma unroll
    for (int d = 0; d < D; ++d) {
        // NaN and values outside end up in the outermost cells
        const float top = (float)((1 << g.bits[d]) - 1);
        c[d] = (uint32_t)fminf(fmaxf((x[d] - g.lo[d]) * g.scale[d], 0.f), top);
        left[d] = g.bits[d];
    }
    uint32_t cell = 0;
    unsigned long long order = g.order;
    for (int s = 0; s < g.steps; ++s, order >>= 2) {
        const int dd = (int)(order & 3u);
        uint32_t bit = 0;
#pragma unroll
        for (int d = 0; d < D; ++d)
            if (d == dd) bit = (c[d] >> --left[d]) & 1u;
        cell = cell * 2u + bit;
    }
    return cell;
}

// Sorted points, box and index arrays carved out of the scratch.
struct SpaceView {
    float4 *pts;                 // sorted points; for d < 4 the index sits in w
    int *idx;                    // index of each sorted point (d = 4)
    float4 *lo[3], *hi[3];       // boxes of leaves, nodes, top entries
    int *mi[3];                  // smallest index in each box
    int n[3];                    // their numbers
    SpaceGrid *grid;
    uint32_t *rank;              // rank of each point in its cell
    uint32_t *block_sum;
    int *far;                    // queries for the brute force
    // cleared together at the start of a call
    uint32_t *bbox;              // [0..3] max ~bits, [4..7] max bits (ordered)
    uint32_t *done;              // blocks of the bounding-box kernel that are done
    int *nfar;                   // length of `far`
    int *crowded;                // a cell holds more than a quarter of the points
    uint32_t *count;             // cells: counts, then first positions
    size_t clear_bytes;
};

// Bounding box of the finite coordinates; the last block to finish lays the
// grid out.
template <int D>
__global__ void __launch_bounds__(256)
    sp_bbox_kernel(const float *__restrict__ ref, int N, long long ldr, int steps, SpaceView v) {
    uint32_t mn[D], mx[D];   // max of the complement, max
#pragma unroll
    for (int d = 0; d < D; ++d) mn[d] = mx[d] = 0u;
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < (unsigned)N; i += gridDim.x * 256)
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const float x = ref[(size_t)d * ldr + i];
            if (isfinite(x)) {
                const uint32_t o = sp_ord(x);
                mn[d] = max(mn[d], ~o);
                mx[d] = max(mx[d], o);
            }
        }
    // one atomic per block and value (per warp they took 42 us at 2^20 points,
    // d = 3; now 6.7)
    __shared__ uint32_t part[8][2 * D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const uint32_t a = __reduce_max_sync(0xffffffffu, mn[d]);
        const uint32_t b = __reduce_max_sync(0xffffffffu, mx[d]);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][d] = a, part[threadIdx.x >> 5][D + d] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2 * D) {
        uint32_t m = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) m = max(m, part[w][threadIdx.x]);
        atomicMax(&v.bbox[threadIdx.x < D ? threadIdx.x : 4 + threadIdx.x - D], m);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(v.done, 1u) == gridDim.x - 1) {
        __threadfence();
        sp_grid<D>(*v.grid, v.bbox, steps);
    }
}

KNN_DI void sp_load_grid(SpaceGrid &g, const SpaceGrid *src) {
    static_assert(sizeof(SpaceGrid) % 4 == 0, "copied in words");
    if (threadIdx.x < sizeof(SpaceGrid) / 4)
        reinterpret_cast<uint32_t *>(&g)[threadIdx.x] =
            reinterpret_cast<const uint32_t *>(src)[threadIdx.x];
    __syncthreads();
}

// Count the points of each cell; a point's rank in its cell is what the counter
// held before its warp's points of that cell, and its place among those.  (An
// atomic for every point serialises where many share a cell: a constant cloud of
// 2^20 points took 440 us here.)
template <int D>
__global__ void __launch_bounds__(256)
    sp_count_kernel(const float *__restrict__ ref, int N, long long ldr, SpaceView v) {
    __shared__ SpaceGrid g;
    sp_load_grid(g, v.grid);
    const int lane = threadIdx.x & 31;
    for (unsigned i0 = blockIdx.x * 256 + (threadIdx.x & ~31u); i0 < (unsigned)N;
         i0 += gridDim.x * 256) {
        const unsigned i = i0 + lane;
        const unsigned in = __ballot_sync(0xffffffffu, i < (unsigned)N);
        if (i >= (unsigned)N) continue;
        float x[D];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = ref[(size_t)d * ldr + i];
        const uint32_t cell = sp_cell<D>(g, x);
        const unsigned same = __match_any_sync(in, cell);
        const int first = __ffs(same) - 1;
        uint32_t rank = 0;
        if (lane == first) rank = atomicAdd(&v.count[cell], (uint32_t)__popc(same));
        rank = __shfl_sync(in, rank, first) + __popc(same & ((1u << lane) - 1u));
        v.rank[i] = rank;
        if (rank == (uint32_t)N / 4) *v.crowded = 1;
    }
}

// Exclusive scan of the cell counters in two kernels: the sum of each block's
// SP_SCAN counters, then each block scans its own on top of the sums before it.
__global__ void __launch_bounds__(256) sp_sum_kernel(SpaceView v, int cells) {
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < SP_SCAN / 256; ++i) {
        const int c = blockIdx.x * SP_SCAN + i * 256 + threadIdx.x;
        if (c < cells) s += v.count[c];
    }
    __shared__ uint32_t part[8];
    s = __reduce_add_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < 8; ++w) t += part[w];
        v.block_sum[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(256) sp_scan_kernel(SpaceView v, int cells) {
    constexpr int PER = SP_SCAN / 256;
    __shared__ uint32_t part[8], before[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the blocks before this one (at most 256 of them)
    uint32_t b = threadIdx.x < blockIdx.x ? v.block_sum[threadIdx.x] : 0u;
    b = __reduce_add_sync(0xffffffffu, b);
    if (lane == 0) before[warp] = b;
    const int c0 = blockIdx.x * SP_SCAN + threadIdx.x * PER;
    uint32_t x[PER], s = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        x[i] = c0 + i < cells ? v.count[c0 + i] : 0u;
        s += x[i];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    uint32_t run = incl - s;
    for (int w = 0; w < 8; ++w) run += before[w] + (w < warp ? part[w] : 0u);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        if (c0 + i < cells) v.count[c0 + i] = run;
        run += x[i];
    }
}

template <int D>
__global__ void __launch_bounds__(256)
    sp_scatter_kernel(const float *__restrict__ ref, int N, long long ldr, SpaceView v) {
    __shared__ SpaceGrid g;
    sp_load_grid(g, v.grid);
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < (unsigned)N; i += gridDim.x * 256) {
        float x[D];
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = ref[(size_t)d * ldr + i];
        const uint32_t pos = v.count[sp_cell<D>(g, x)] + v.rank[i];
        float4 p = make_float4(x[0], D > 1 ? x[1 % D] : 0.f, D > 2 ? x[2 % D] : 0.f,
                               D > 3 ? x[3 % D] : __uint_as_float(i));
        v.pts[pos] = p;
        if (D == 4) v.idx[pos] = (int)i;
    }
}

// Box of the 32 lanes' boxes [lo, hi] (NaN coordinates take no part).
template <int D>
KNN_DI void sp_warp_box(float (&lo)[4], float (&hi)[4], int &mi) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const bool nan = !(lo[d] == lo[d]) || !(hi[d] == hi[d]);
        const uint32_t a = __reduce_min_sync(0xffffffffu, nan ? 0xffffffffu : sp_ord(lo[d]));
        const uint32_t b = __reduce_max_sync(0xffffffffu, nan ? 0u : sp_ord(hi[d]));
        // no coordinate at all: an empty box, infinitely far from everything
        lo[d] = a == 0xffffffffu ? INFINITY : sp_unord(a);
        hi[d] = b == 0u ? -INFINITY : sp_unord(b);
    }
    mi = (int)__reduce_min_sync(0xffffffffu, (unsigned)mi);
}

template <int D>
KNN_DI void sp_store_box(const SpaceView &v, int level, int i, const float (&lo)[4],
                         const float (&hi)[4], int mi) {
    v.lo[level][i] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    v.hi[level][i] = make_float4(hi[0], hi[1], hi[2], hi[3]);
    v.mi[level][i] = mi;
}

// One block per node: a warp per leaf, then the node from its leaves.
template <int D>
__global__ void __launch_bounds__(1024) sp_leaf_kernel(SpaceView v, int N) {
    __shared__ float slo[32][4], shi[32][4];
    __shared__ int smi[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int leaf = blockIdx.x * 32 + warp, i = leaf * 32 + lane;
    float lo[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
    float hi[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    int mi = 0x7fffffff;
    if (i < N) {
        const float4 p = v.pts[i];
        lo[0] = hi[0] = p.x;
        if (D > 1) lo[1] = hi[1] = p.y;
        if (D > 2) lo[2] = hi[2] = p.z;
        if (D > 3) lo[3] = hi[3] = p.w;
        mi = D == 4 ? v.idx[i] : __float_as_int(p.w);
    }
    sp_warp_box<D>(lo, hi, mi);
    if (lane == 0) {
        if (leaf < v.n[0]) sp_store_box<D>(v, 0, leaf, lo, hi, mi);
#pragma unroll
        for (int d = 0; d < 4; ++d) slo[warp][d] = lo[d], shi[warp][d] = hi[d];
        smi[warp] = mi;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int d = 0; d < 4; ++d) lo[d] = slo[lane][d], hi[d] = shi[lane][d];
        mi = smi[lane];
        sp_warp_box<D>(lo, hi, mi);
        if (lane == 0) sp_store_box<D>(v, 1, blockIdx.x, lo, hi, mi);
    }
}

// A warp per top entry, from its nodes.
template <int D>
__global__ void __launch_bounds__(128) sp_top_kernel(SpaceView v) {
    const int top = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (top >= v.n[2]) return;
    const int c = top * 32 + lane;
    float lo[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
    float hi[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    int mi = 0x7fffffff;
    if (c < v.n[1]) {
        const float4 a = v.lo[1][c], b = v.hi[1][c];
        lo[0] = a.x; lo[1] = a.y; lo[2] = a.z; lo[3] = a.w;
        hi[0] = b.x; hi[1] = b.y; hi[2] = b.z; hi[3] = b.w;
        mi = v.mi[1][c];
    }
    sp_warp_box<D>(lo, hi, mi);
    if (lane == 0) sp_store_box<D>(v, 2, top, lo, hi, mi);
}

// Lower bound (distance bits << 32 | smallest index) of box i of a level: not
// above the key of any point in it.  kKeyInf beyond the level and for boxes
// infinitely far away.
template <int D>
KNN_DI unsigned long long sp_bound(const SpaceView &v, int level, int i, int n,
                                   const float (&q)[D]) {
    if (i >= n) return kKeyInf;
    const float4 a = v.lo[level][i], b = v.hi[level][i];
    const float lo[4] = {a.x, a.y, a.z, a.w}, hi[4] = {b.x, b.y, b.z, b.w};
    float acc = 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const float t = fmaxf(fmaxf(__fsub_rn(lo[d], q[d]), __fsub_rn(q[d], hi[d])), 0.f);
        acc = __fmaf_rn(t, t, acc);
    }
    return finite_key(acc, (uint32_t)v.mi[level][i]);
}

// One warp per query.
template <int D>
__global__ void __launch_bounds__(32 * SP_WARPS)
    sp_search_kernel(const float *__restrict__ qry, int Q, long long ldq, int N, int k, int cap,
                     SpaceView v, float *__restrict__ out_dist, int *__restrict__ out_idx,
                     long long ld_out) {
    __shared__ SpaceGrid g;
    sp_load_grid(g, v.grid);
    const int lane = threadIdx.x & 31;
    // (unsigned: the last block's queries may lie beyond the largest int)
    const unsigned qi = blockIdx.x * SP_WARPS + (threadIdx.x >> 5);
    if (qi >= (unsigned)Q) return;
    float q[D];
    bool finite = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        q[d] = qry[(size_t)d * ldq + qi];
        finite = finite && isfinite(q[d]);
    }
    // lane j holds the j-th smallest key; tau is the k-th
    unsigned long long mine = kKeyNone, tau = kKeyNone;
    int visits = 0;
    auto leaf_scan = [&](int leaf) {
        const int i = leaf * 32 + lane;
        unsigned long long key = kKeyInf;
        if (i < N) {
            const float4 p = v.pts[i];
            const float x[4] = {p.x, p.y, p.z, p.w};
            float acc = 0.f;
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const float t = __fsub_rn(x[d], q[d]);
                acc = __fmaf_rn(t, t, acc);
            }
            const int id = D == 4 ? v.idx[i] : __float_as_int(p.w);
            key = finite_key(acc, (uint32_t)id);
        }
        ++visits;
        lane_list_add(mine, tau, key, k, lane);
    };
    // the lane with the smallest bound below tau among those still open
    auto nearest = [&](unsigned long long &b) {
        const uint32_t h = (uint32_t)(b >> 32);
        const uint32_t mn = __reduce_min_sync(0xffffffffu, b < tau ? h : 0xffffffffu);
        if (mn == 0xffffffffu) return -1;
        const int c = __ffs(__ballot_sync(0xffffffffu, b < tau && h == mn)) - 1;
        if (lane == c) b = kKeyInf;
        return c;
    };
    if (finite && *v.crowded) {
        visits = cap + 1;
    } else if (finite) {
        const uint32_t at = v.count[sp_cell<D>(g, q)];
        const int first = (int)min(at, (uint32_t)(N - 1)) / 32;
        leaf_scan(first);
        for (int t0 = 0; t0 < v.n[2] && visits <= cap; t0 += 32) {
            unsigned long long bt = sp_bound<D>(v, 2, t0 + lane, v.n[2], q);
            for (int ct; visits <= cap && (ct = nearest(bt)) >= 0;) {
                const int node0 = (t0 + ct) * 32;
                unsigned long long bn = sp_bound<D>(v, 1, node0 + lane, v.n[1], q);
                for (int cn; visits <= cap && (cn = nearest(bn)) >= 0;) {
                    const int leaf0 = (node0 + cn) * 32;
                    unsigned long long bl = sp_bound<D>(v, 0, leaf0 + lane, v.n[0], q);
                    if (leaf0 + lane == first) bl = kKeyInf;
                    for (int cl; visits <= cap && (cl = nearest(bl)) >= 0;) leaf_scan(leaf0 + cl);
                }
            }
        }
    }
    if (visits > cap) {
        if (lane == 0) v.far[atomicAdd(v.nfar, 1)] = (int)qi;
        return;
    }
    if (lane < k) {
        out_dist[(size_t)lane * ld_out + qi] = sqrtf(key_dist2(mine));
        out_idx[(size_t)lane * ld_out + qi] = key_index(mine);
    }
}

int sp_steps(int N) {
    int b = 1;
    while (b < SP_MAX_BITS && (1 << b) < N) ++b;
    return b;
}

size_t sp_carve(SpaceView &v, void *mem, int N, int Q, int d) {
    unsigned char *p = static_cast<unsigned char *>(mem);
    size_t used = 0;
    auto take = [&](size_t bytes) {
        void *r = p ? p + used : nullptr;
        used += (bytes + 255) / 256 * 256;
        return r;
    };
    v.n[0] = (N + 31) / 32;
    v.n[1] = (v.n[0] + 31) / 32;
    v.n[2] = (v.n[1] + 31) / 32;
    v.pts = static_cast<float4 *>(take((size_t)N * 16));
    v.idx = static_cast<int *>(take(d == 4 ? (size_t)N * 4 : 0));
    for (int l = 0; l < 3; ++l) {
        v.lo[l] = static_cast<float4 *>(take((size_t)v.n[l] * 16));
        v.hi[l] = static_cast<float4 *>(take((size_t)v.n[l] * 16));
        v.mi[l] = static_cast<int *>(take((size_t)v.n[l] * 4));
    }
    v.grid = static_cast<SpaceGrid *>(take(sizeof(SpaceGrid)));
    v.rank = static_cast<uint32_t *>(take((size_t)N * 4));
    v.block_sum = static_cast<uint32_t *>(take(256 * 4));
    v.far = static_cast<int *>(take((size_t)Q * 4));
    const size_t cleared = used;
    v.bbox = static_cast<uint32_t *>(take(8 * 4));
    v.done = static_cast<uint32_t *>(take(4));
    v.nfar = static_cast<int *>(take(4));
    v.crowded = static_cast<int *>(take(4));
    v.count = static_cast<uint32_t *>(take(sizeof(uint32_t) << sp_steps(N)));
    v.clear_bytes = used - cleared;
    return used;
}

template <int D>
int launch_space_d(const ExactProblem &p, const SpaceView &v, cudaStream_t st) {
    const int steps = sp_steps(p.N), cells = 1 << steps;
    const int blocks = std::min((p.N + 255) / 256, 8 * p.num_sms);
    if (cudaMemsetAsync(v.bbox, 0, v.clear_bytes, st) != cudaSuccess) return kErrCuda;
    sp_bbox_kernel<D><<<blocks, 256, 0, st>>>(p.ref, p.N, p.ldr, steps, v);
    sp_count_kernel<D><<<blocks, 256, 0, st>>>(p.ref, p.N, p.ldr, v);
    const int sb = (cells + SP_SCAN - 1) / SP_SCAN;
    sp_sum_kernel<<<sb, 256, 0, st>>>(v, cells);
    sp_scan_kernel<<<sb, 256, 0, st>>>(v, cells);
    sp_scatter_kernel<D><<<blocks, 256, 0, st>>>(p.ref, p.N, p.ldr, v);
    sp_leaf_kernel<D><<<v.n[1], 1024, 0, st>>>(v, p.N);
    sp_top_kernel<D><<<(v.n[2] + 3) / 4, 128, 0, st>>>(v);
    const int cap = std::max(256, v.n[0] / 64);
    sp_search_kernel<D><<<(unsigned)(((long long)p.Q + SP_WARPS - 1) / SP_WARPS), 32 * SP_WARPS,
                          0, st>>>(
        p.qry, p.Q, p.ldq, p.N, p.k, cap, v, p.out_dist, p.out_idx, p.ld_out);
    return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

}  // namespace

bool space_applies(int N, int Q, int d, int k) {
    // Ordering the points costs about 35 us and 45 us per 2^20 of them, a search
    // about as much as 1000 to 2500 pairs of the brute force.  Brute force / search
    // in us at d = 1, k = 8 and at d = 4, k = 16: 33 / 48 and 45 / 82 with 10000 x
    // 1000, 56 / 48 and 90 / 87 with 7000 x 7000, 73 / 50 and 116 / 91 with 25000 x
    // 2000, 71 / 79 and 101 / 189 with 2^20 x 50, 173 / 100 and 256 / 197 with 2^20 x
    // 200, 736 / 82 and 1449 / 195 with 2^20 x 1600.
    // A search never costs less than about 0.6 us a thousand queries (d = 1, k = 1; 1.9
    // at d = 4, k = 16), so few points are searched by brute force however many the
    // queries are: 831 / 1297 with 512 x 10^6 at d = 3, k = 8, 1258 / 1349 with 1000 x
    // 10^6 (1846 / 1351 where the points are sorted); in one dimension 498 / 694 with
    // 256 x 10^6, 791 / 720 with 512 x 10^6 (k = 8).
    return d >= 1 && d <= 4 && k >= 1 && k <= 16 && N <= (1 << 30) &&
           (double)N * Q >= 5e7 + 100.0 * N && N >= (d == 1 ? 400 : 700);
}

size_t space_bytes(int N, int Q, int d, int k) {
    if (!space_applies(N, Q, d, k)) return 0;
    SpaceView v;
    return sp_carve(v, nullptr, N, Q, d);
}

int launch_space(const ExactProblem &p, cudaStream_t st, QuerySubset *far) {
    SpaceView v;
    if (!p.space || sp_carve(v, p.space, p.N, p.Q, p.d) > p.space_bytes) return kErrScratch;
    far->list = v.far;
    far->count = v.nfar;
    switch (p.d) {
        case 1: return launch_space_d<1>(p, v, st);
        case 2: return launch_space_d<2>(p, v, st);
        case 3: return launch_space_d<3>(p, v, st);
        default: return launch_space_d<4>(p, v, st);
    }
}

}  // namespace knnb200
