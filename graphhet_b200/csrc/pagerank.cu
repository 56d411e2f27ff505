// PageRank, pull form over the in-CSR (replaces GPU_PR_csr.cuh:34-197;
// semantics of CPU_PageRank.hpp:12-56):
//   S       = sum of rank[u] over vertices with no out-edges
//   rank'[v] = (1-d)/N + d*S/N + d * sum_{u in in(v)} rank[u] / outdeg(u)
//
// Per iteration one pass reads in_rowptr and in_col once and gathers
// contrib[u] = rank[u] / outdeg(u) (precomputed once per vertex, so the
// per-entry division of the CPU path becomes a per-vertex one with the same
// FP64 result).  The same pass writes rank' and the next contrib, and block
// partials of the next S and of the L1 change; a one-block kernel reduces the
// partials in a fixed order (deterministic S and norm, FP64 in both modes).
//
// The non-empty rows' entries are cut into tiles of 256, a warp each; rows that
// cross tiles are combined in tile order.  The hubs' contributions come from a
// shared-memory cache (a degree-relabelled graph puts the hubs first).
//
// FP32 mode: ranks and contributions are stored as float (half the gather
// footprint: 64 MiB at n = 2^24, resident in the 126 MB L2); each lane keeps
// a Kahan-compensated FP32 sum and lanes are merged with an error-free
// TwoSum; the row total, S and the L1 norm are FP64.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "scan.cuh"

namespace ghb {
namespace {

constexpr int kPrThreads = 256;

template <class T>
struct KSum;  // per-lane accumulator

template <>
struct KSum<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double x) { s += x; }
    __device__ __forceinline__ void merge_from_lane(int offset, int width) {
        s += __shfl_down_sync(0xffffffffu, s, offset, width);
    }
    __device__ __forceinline__ double value() const { return s; }
};

template <>
struct KSum<float> {
    float s = 0.f, c = 0.f;  // true sum ~= s - c
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ void merge_from_lane(int offset, int width) {
        const float s2 = __shfl_down_sync(0xffffffffu, s, offset, width);
        const float c2 = __shfl_down_sync(0xffffffffu, c, offset, width);
        // TwoSum: t + err == s + s2 exactly.
        const float t = s + s2;
        const float bp = t - s;
        const float err = (s - (t - bp)) + (s2 - bp);
        s = t;
        c = c + c2 - err;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

template <class T>
__device__ __forceinline__ T load_contrib(const T* p, uint64_t pol);
template <>
__device__ __forceinline__ double load_contrib<double>(const double* p, uint64_t pol) {
    return ld_keep_f64(p, pol);
}
template <>
__device__ __forceinline__ float load_contrib<float>(const float* p, uint64_t pol) {
    return ld_keep_f32(p, pol);
}

struct PrScalars {
    double base;  // (1-d)/N + d*S/N for the current iteration
    double l1;    // L1 change of the last iteration
    double sink;  // S of the current ranks
};

// rank0 = 1/N, contrib0 = rank0/outdeg, block partials of S0.
template <class T>
__global__ void __launch_bounds__(kPrThreads) pr_init_kernel(int32_t n, const int32_t* __restrict__ out_rp,
                                                             int32_t* __restrict__ outdeg, T* rank,
                                                             T* contrib, T* contrib_next, double* part_sink) {
    __shared__ double red[kPrThreads / 32];
    double sink = 0.0;
    const double r0 = 1.0 / (double)n;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = out_rp[v + 1] - out_rp[v];
        outdeg[v] = d;
        rank[v] = (T)r0;
        contrib[v] = d > 0 ? (T)(r0 / (double)d) : (T)0;
        contrib_next[v] = (T)0;  // an isolated vertex's is not written again
        if (d == 0) sink += (double)(T)r0;
    }
    sink = warp_sum(sink);
    if (lane_id() == 0) red[threadIdx.x >> 5] = sink;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < kPrThreads / 32; ++i) s += red[i];
        part_sink[blockIdx.x] = s;
    }
}

template <class T>
__device__ __forceinline__ void pr_finish_row(int64_t v, int32_t d, double sum, double base, double damping,
                                              const T* rank_old, T* rank_new, T* contrib_new, int track_l1,
                                              double& sink, double& l1) {
    const double r = base + damping * sum;
    const T rt = (T)r;
    rank_new[v] = rt;
    contrib_new[v] = d > 0 ? (T)(r / (double)d) : (T)0;
    if (d == 0) sink += (double)rt;
    if (track_l1) l1 += fabs((double)rt - (double)rank_old[v]);
}

template <class T>
__device__ __forceinline__ void block_partials(double sink, double l1, double* part_sink, double* part_l1,
                                               int slot) {
    __shared__ double red_s[32], red_l[32];
    sink = warp_sum(sink);
    l1 = warp_sum(l1);
    if (lane_id() == 0) {
        red_s[threadIdx.x >> 5] = sink;
        red_l[threadIdx.x >> 5] = l1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0, l = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            s += red_s[i];
            l += red_l[i];
        }
        part_sink[slot] = s;
        part_l1[slot] = l;
    }
}

// Shared-memory cache of the first K contributions (K from the workspace's
// pr_cache_kb).  On a degree-relabelled graph these are the hubs' (the top 10 K
// vertices of an RMAT scale-22 graph hold a third of all entries), so their
// gathers take no L2 sector.  The kernel runs persistent blocks (pr_threads x
// pr_blocks_per_sm per SM, 1024 x 1 by default), so each fills the cache once
// per launch.
constexpr int kPrPersistThreads = 1024;
// The most that a block may ask for beside its static words.
constexpr int kPrMaxSmem = 226 * 1024;

template <class T>
__device__ __forceinline__ int32_t fill_hub_cache(T* cache, const T* __restrict__ contrib_old, int32_t n,
                                                  int32_t cache_elems) {
    const int32_t K = min(cache_elems, n);
    for (int32_t i = threadIdx.x; i < K; i += blockDim.x) cache[i] = contrib_old[i];
    __syncthreads();
    return K;
}

template <class T>
__device__ __forceinline__ T gather(const T* cache, int32_t K, const T* __restrict__ contrib_old, int32_t u,
                                    uint64_t pol) {
    return u < K ? cache[u] : load_contrib<T>(contrib_old + u, pol);
}

// One block: S and L1 from the partials (fixed order), next base.
__device__ __forceinline__ void pr_reduce(const double* part_sink, const double* part_l1, int nparts, int32_t n,
                                          double damping, PrScalars* sc, double* l1_hist, int iter, int has_l1) {
    __shared__ double rs[kPrThreads], rl[kPrThreads];
    double s = 0.0, l = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        s += __ldcg(part_sink + i);
        if (has_l1) l += __ldcg(part_l1 + i);
    }
    rs[threadIdx.x] = s;
    rl[threadIdx.x] = l;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            rs[threadIdx.x] += rs[threadIdx.x + o];
            rl[threadIdx.x] += rl[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double S = rs[0];
        sc->sink = S;
        sc->base = (1.0 - damping) / (double)n + S * damping / (double)n;
        if (has_l1) {
            sc->l1 = rl[0];
            if (l1_hist) l1_hist[iter] = rl[0];
        }
    }
}
__global__ void __launch_bounds__(kPrThreads) pr_reduce_kernel(const double* part_sink, const double* part_l1,
                                                               int nparts, int32_t n, double damping, PrScalars* sc) {
    pr_reduce(part_sink, part_l1, nparts, n, damping, sc, nullptr, 0, 0);
}

// ---- tiles
//
// The entries of the non-empty rows, taken in order, are cut into tiles of
// kPrTile; a warp takes a tile, whatever rows it holds.  So every warp has the
// same number of gathers, all of them in flight at once, where a thread per
// short row left a third of the lanes idle and its blocks uneven, and rows cut
// into chunks needed kernels of their own.  A tile inside one row is summed in
// registers; in a mixed one the values go through the warp's shared memory and
// each row's are summed by a lane (by the warp from 32 values on).  A row that
// crosses tiles leaves a partial sum per tile: tail[t] in the tile where it
// begins, head[t] in those that it continues into; pr_finish_kernel adds them in
// tile order, so results do not depend on timing.
constexpr int kPrPerLane = 8;
constexpr int32_t kPrTile = 32 * kPrPerLane;

// Non-empty rows in ascending order: row ids and their first entries (begin[k]
// = m behind the last; only the device knows how many rows there are).
struct PrRows {
    const int32_t* __restrict__ id;     // id[i]
    const int32_t* __restrict__ begin;  // begin[i], begin[k] = m
    const int32_t* __restrict__ deg;    // out-degrees
    const int32_t* __restrict__ tile;   // tile[t]: the row (index) that holds entry t * kPrTile; tile[tiles]: the last
    int32_t m;
    int32_t tiles;
};

__global__ void pr_row_flags_kernel(int32_t n, const int32_t* __restrict__ in_rp, int32_t* flag) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        flag[v] = in_rp[v + 1] > in_rp[v] ? 1 : 0;
}

// pos = exclusive scan of the flags: the non-empty rows' ids, offsets and
// out-degrees in order.  Rows without entries go to `bare`, those with
// out-entries from the front, isolated ones from the back; count[0], count[1].
__global__ void __launch_bounds__(256) pr_row_lists_kernel(int32_t n, const int32_t* __restrict__ in_rp,
                                                           const int32_t* __restrict__ pos,
                                                           const int32_t* __restrict__ outdeg, int32_t* id,
                                                           int32_t* begin, int32_t* deg, int32_t* bare,
                                                           int32_t* count) {
    __shared__ int32_t s_n[2], s_at[2];
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x; v0 < n; v0 += (int64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
        __syncthreads();
        const int64_t v = v0 + threadIdx.x;
        int kind = -1;
        int32_t at = 0;
        if (v < n) {
            const int32_t b = in_rp[v], d = outdeg[v];
            if (in_rp[v + 1] > b) {
                const int32_t i = pos[v];
                id[i] = (int32_t)v;
                begin[i] = b;
                deg[i] = d;
            } else {
                kind = d > 0 ? 0 : 1;
                at = atomicAdd(&s_n[kind], 1);
            }
            if (v == n - 1) begin[pos[n]] = in_rp[n];
        }
        __syncthreads();
        if (threadIdx.x < 2 && s_n[threadIdx.x]) s_at[threadIdx.x] = atomicAdd(count + threadIdx.x, s_n[threadIdx.x]);
        __syncthreads();
        if (kind == 0) bare[s_at[0] + at] = (int32_t)v;
        if (kind == 1) bare[n - 1 - (s_at[1] + at)] = (int32_t)v;
        __syncthreads();
    }
}

__global__ void pr_tile_rows_kernel(const int32_t* __restrict__ rows, const int32_t* __restrict__ begin, int32_t tiles,
                                    int32_t* tile) {
    const int32_t k = *rows;
    if (blockIdx.x == 0 && threadIdx.x == 0) tile[tiles] = k - 1;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tiles; t += (int64_t)gridDim.x * blockDim.x) {
        int32_t lo = 0, hi = k - 1;  // the last row that begins at or before the entry
        while (lo < hi) {
            const int32_t mid = (int32_t)(((int64_t)lo + hi + 1) >> 1);
            if ((int64_t)begin[mid] <= t * kPrTile) lo = mid;
            else hi = mid - 1;
        }
        tile[t] = lo;
    }
}

template <class T>
__device__ __forceinline__ double warp_total(KSum<T> acc) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc.merge_from_lane(o, 32);
    return __shfl_sync(0xffffffffu, acc.value(), 0);
}

// Bound by the gathers: each takes a 32-byte sector of L2 or its own pass of
// the L1 pipe, which is busy 82 % of the time (L2 58 %, DRAM 18 %; directed RMAT of
// 2^23 vertices and 83 M entries, FP64).  12 M vertices, 160 M entries, FP64: 0.61 ms an iteration (260 G
// gathers/s), where a thread per short row and a warp per chunk of a longer one
// took 0.35 + 0.49 ms.  Tiles and entries are counted in 32 bits (there are
// fewer than 2^31): in 64 the kernel spilled, 0.68 ms.  Ten iterations in all
// 7.0 ms with 256 entries a tile, 7.1 with 224, 7.4 with 160 or 320 (spills).
template <class T>
__global__ void __launch_bounds__(kPrPersistThreads) pr_tile_kernel(
    PrRows R, int32_t n, const int32_t* __restrict__ in_col, const T* __restrict__ contrib_old, const T* rank_old,
    T* rank_new, T* contrib_new, const PrScalars* sc, double damping, int track_l1, double* head, double* tail, double* part_sink, double* part_l1,
    int32_t cache_elems) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* cache = reinterpret_cast<T*>(smem_raw);
    T* vals = cache + ((cache_elems + 3) & ~3) + (threadIdx.x >> 5) * kPrTile;
    const int32_t K = fill_hub_cache<T>(cache, contrib_old, n, cache_elems);
    const uint64_t pol_stream = policy_evict_first();
    const uint64_t pol_keep = policy_evict_last();
    const int lane = lane_id();
    const int32_t warp = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int32_t nwarps = (int32_t)((gridDim.x * blockDim.x) >> 5);
    double sink = 0.0, l1 = 0.0;
    const double base = sc->base;
    auto finish = [&](int32_t row, int32_t d, double sum) {
        pr_finish_row<T>(row, d, sum, base, damping, rank_old, rank_new, contrib_new, track_l1, sink, l1);
    };
    // A tile is a chain of columns, gathers and writes; the next tile's columns
    // and this tile's row data are loaded under the gathers.
    auto load_cols = [&](int32_t t, int32_t (&u)[kPrPerLane]) {
        const uint32_t t0 = (uint32_t)t * kPrTile;
#pragma unroll
        for (int q = 0; q < kPrPerLane; ++q)
            u[q] = t0 + q * 32 + lane < (uint32_t)R.m ? ld_stream(in_col + t0 + q * 32 + lane, pol_stream) : -1;
    };
    int32_t ahead[kPrPerLane];
    int32_t ahead0 = 0, ahead1 = 0;
    if (warp < R.tiles) {
        load_cols(warp, ahead);
        ahead0 = R.tile[warp];
        ahead1 = R.tile[warp + 1];
    }
    for (int32_t t = warp; t < R.tiles; t += nwarps) {
        const uint32_t t0 = (uint32_t)t * kPrTile, t1 = min(t0 + kPrTile, (uint32_t)R.m);
        T x[kPrPerLane];
        unsigned ok = 0;
#pragma unroll
        for (int q = 0; q < kPrPerLane; ++q) {
            x[q] = ahead[q] >= 0 ? gather<T>(cache, K, contrib_old, ahead[q], pol_keep) : (T)0;
            ok |= ahead[q] >= 0 ? 1u << q : 0u;
        }
        const int32_t i0 = ahead0, i1 = ahead1;
        int32_t i = i0 + lane, b = 0, e = 0, id = 0, deg = 0;
        auto load_row = [&]() {
            b = e = 0;
            if (i <= i1) {
                b = R.begin[i];
                e = R.begin[i + 1];
                id = R.id[i];
                deg = R.deg[i];
            }
        };
        load_row();
        if (t + nwarps < R.tiles) {
            load_cols(t + nwarps, ahead);
            ahead0 = R.tile[t + nwarps];
            ahead1 = R.tile[t + nwarps + 1];
        }
        if ((uint32_t)__shfl_sync(0xffffffffu, e, 0) >= t1) {  // one row
            KSum<T> acc;
#pragma unroll
            for (int q = 0; q < kPrPerLane; ++q)
                if ((ok >> q) & 1u) acc.add(x[q]);
            const double v = warp_total(acc);
            if (lane == 0) {
                if ((uint32_t)b < t0) head[t] = v;
                else if ((uint32_t)e > t1) tail[t] = v;
                else finish(id, deg, v);
            }
            continue;
        }
#pragma unroll
        for (int q = 0; q < kPrPerLane; ++q) vals[q * 32 + lane] = x[q];
        __syncwarp();
        while (true) {
            const int32_t s = (int32_t)(max((uint32_t)b, t0) - t0);
            const int32_t len = i <= i1 ? (int32_t)(min((uint32_t)e, t1) - t0) - s : 0;  // 0 or less: the next tile's row
            double v = 0.0;
            if (len > 0 && len < 32) {
                KSum<T> acc;
                for (int32_t j = s; j < s + len; ++j) acc.add(vals[j]);
                v = acc.value();
            }
            unsigned longer = __ballot_sync(0xffffffffu, len >= 32);
            while (longer) {
                const int l = __ffs(longer) - 1;
                longer &= longer - 1;
                const int32_t ls = __shfl_sync(0xffffffffu, s, l), ll = __shfl_sync(0xffffffffu, len, l);
                KSum<T> acc;
                for (int32_t j = lane; j < ll; j += 32) acc.add(vals[ls + j]);
                const double w = warp_total(acc);
                if (lane == l) v = w;
            }
            if (len > 0) {
                if ((uint32_t)b < t0) head[t] = v;
                else if ((uint32_t)e > t1) tail[t] = v;
                else finish(id, deg, v);
            }
            i += 32;
            if (__shfl_sync(0xffffffffu, i, 0) > i1) break;
            load_row();
        }
        __syncwarp();
    }
    block_partials<T>(sink, l1, part_sink, part_l1, blockIdx.x);
}

// The rows that cross tiles (a thread per tile in which one begins; the warp
// together where it spans more than kPrSpan) and the rows without entries, whose
// rank is the base: isolated ones pass nothing on, so until the last iteration
// only their share of S is counted (all: every row, when the change is tracked
// or ranks are due).  Then, in the
// block that ends last, S and L1 from all blocks' partials in a fixed order and
// the next base.
constexpr int64_t kPrSpan = 16;
template <class T>
__global__ void __launch_bounds__(kPrThreads) pr_finish_kernel(
    PrRows R, int32_t n, const int32_t* __restrict__ bare, const int32_t* __restrict__ bare_count, int all,
    const double* __restrict__ head,
    const double* __restrict__ tail, const int32_t* __restrict__ outdeg, const T* rank_old, T* rank_new,
    T* contrib_new, PrScalars* sc, double damping, int track_l1, double* part_sink, double* part_l1, int slot0,
    int nparts, double* l1_hist, int iter, int32_t* done) {
    const int lane = lane_id();
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nt = (int64_t)gridDim.x * blockDim.x;
    const double base = sc->base;
    double sink = 0.0, l1 = 0.0;
    for (int64_t tb = tid - lane; tb < R.tiles; tb += nt) {
        const int64_t t = tb + lane;
        int32_t row = -1, deg = 0;
        int64_t last = 0;
        if (t < R.tiles) {
            // The tile's last row crosses its end when it holds the next tile's
            // first entry as well, and begins here unless it began before.
            const int32_t i = R.tile[t + 1];
            const int64_t b = R.begin[i], e = R.begin[i + 1];
            if (b >= t * kPrTile && b < (t + 1) * kPrTile && e > (t + 1) * kPrTile) {
                row = R.id[i];
                deg = R.deg[i];
                last = (e - 1) / kPrTile;
            }
        }
        double sum = 0.0;
        if (row >= 0 && last - t <= kPrSpan) {
            sum = tail[t];
            for (int64_t x = t + 1; x <= last; ++x) sum += head[x];
        }
        unsigned wide = __ballot_sync(0xffffffffu, row >= 0 && last - t > kPrSpan);
        while (wide) {
            const int l = __ffs(wide) - 1;
            wide &= wide - 1;
            const int64_t t2 = tb + l, last2 = __shfl_sync(0xffffffffu, last, l);
            double s = lane == 0 ? tail[t2] : 0.0;
            for (int64_t x = t2 + 1 + lane; x <= last2; x += 32) s += head[x];
            s = warp_sum(s);
            if (lane == l) sum = s;
        }
        if (row >= 0)
            pr_finish_row<T>(row, deg, sum, base, damping, rank_old, rank_new, contrib_new, track_l1, sink, l1);
    }
    const int32_t with_out = bare_count[0], isolated = bare_count[1];
    for (int64_t i = tid; i < with_out; i += nt)
        pr_finish_row<T>(bare[i], outdeg[bare[i]], 0.0, base, damping, rank_old, rank_new, contrib_new, track_l1, sink,
                         l1);
    if (all) {
        for (int64_t i = tid; i < isolated; i += nt)
            pr_finish_row<T>(bare[n - 1 - i], 0, 0.0, base, damping, rank_old, rank_new, contrib_new, track_l1, sink, l1);
    } else if (tid == 0) {
        sink += (double)(T)base * (double)isolated;
    }
    block_partials<T>(sink, l1, part_sink, part_l1, slot0 + blockIdx.x);
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1) == (int32_t)gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    if (threadIdx.x == 0) *done = 0;
    pr_reduce(part_sink, part_l1, nparts, n, damping, sc, l1_hist, iter, track_l1);
}

// The ranks to the caller, through perm where the rows are in other ids.
template <class T>
__global__ void pr_to_f64_kernel(const T* __restrict__ src, const int32_t* __restrict__ perm, double* dst, int32_t n) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x)
        dst[v] = (double)src[perm ? perm[v] : v];
}

template <class T>
int pagerank_impl(ghb_workspace* ws, int32_t n, int64_t m, const int32_t* in_rp, const int32_t* in_col,
                  const int32_t* out_rp, const ghb_pr_options* o, double* rank_out, int32_t* iters_run, const int32_t* perm) {
    const bool ranked = perm != nullptr;
    cudaStream_t st = ws->stream;
    int32_t* hp = reinterpret_cast<int32_t*>(ws->host_pinned);
    // Not to be recorded: a later call may move the scratch that a graph would
    // replay on.
    cudaStreamCaptureStatus recording;
    GHB_CUDA_TRY(cudaStreamIsCapturing(st, &recording));
    if (recording != cudaStreamCaptureStatusNone) {
        set_error("PageRank: operation not permitted when the stream is capturing");
        return GHB_ERR_CUDA;
    }
    if (m < 0) {
        GHB_CUDA_TRY(cudaMemcpyAsync(hp, in_rp + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        GHB_CUDA_TRY(cudaStreamSynchronize(st));
        m = hp[0];
    }
    const Tuning& tu = ws->tune;
    // A small graph's few tiles spread over more blocks, without a cache that each
    // would have to fill.  An iteration with a look at the change, 1,024 threads and
    // 16 KB against these: 120 k entries 42.4 and 36.5 us, 200 k 42.7 and 35.5, 430 k
    // 42.0 and 36.5; 8 k without the look 14.5 and 12.5.  From 2^20 entries on wider
    // blocks are as good or better (2.4 M 28.7, 30.8 with 512, 35.8 with 256).
    const int pthreads = std::min(tu.pr_threads, m < (1 << 18) ? 256 : m < (1 << 20) ? 512 : kPrPersistThreads);
    const unsigned max_rows = ws->num_sms * tu.pr_blocks_per_sm;  // persistent blocks
    // Hub cache and the warps' tiles share a block's shared memory.
    const size_t tile_bytes = (size_t)(pthreads / 32) * kPrTile * sizeof(T);
    const size_t block_smem = (size_t)(227 * 1024) / tu.pr_blocks_per_sm - (tu.pr_blocks_per_sm > 1 ? 1024 : 0);
    // Shared memory taken from L1 costs more than it gives past some 96 KB (160 M
    // entries, FP64, ten iterations: 8.3 ms without a cache, 7.8 with 64 to 96 KB,
    // 8.4 with 112, 13.1 with 144), and where the first ids are not the hubs
    // nothing is gained from 32 KB on (9.7 ms with 0 or 32 KB, 10.8 with 64).
    // Below 2^24 entries a block gathers too little for its fill (and below 2^20 for
    // any; ten iterations with 16 and 80 KB: 2 M entries 306 and 332 us, 8 M 485 and 498; with 32 M
    // 1,260 and 1,220).
    const int32_t most_kb = m < (1 << 20) ? 0 : m < (1 << 24) ? 16 : ranked ? tu.pr_cache_kb : 32;
    const int32_t cache_kb = std::min(tu.pr_cache_kb, most_kb);
    const size_t cache_bytes = std::min((size_t)cache_kb * 1024,
                                        block_smem > tile_bytes + 1024 ? (block_smem - tile_bytes - 1024) & ~(size_t)255 : 0);
    const int32_t cache_elems = (int32_t)(cache_bytes / sizeof(T));
    const size_t smem = (size_t)((cache_elems + 3) & ~3) * sizeof(T) + tile_bytes;
    const int32_t tiles = (int32_t)((m + kPrTile - 1) / kPrTile);
    const unsigned grid_rows = tiles ? grid_for((int64_t)tiles * 32, pthreads, max_rows) : 0;
    const unsigned grid_fin = grid_for(std::max<int64_t>(tiles, n / 8), kPrThreads, ws->num_sms * 8);
    const int nparts = (int)(grid_rows + grid_fin);
    const unsigned g = ws->num_sms * 8;
    const unsigned grid_init = grid_for(n, kPrThreads, nparts);  // one partial slot per block
    T *ra, *rb, *ca, *cb;
    int32_t *outdeg, *flag, *pos, *row_id, *row_begin, *row_deg, *bare, *bare_count, *tile, *done;
    double *head, *tail, *ps, *pl, *hist;
    int64_t* bs;
    PrScalars* sc;
    auto carve = [&](Carver& c) {
        ra = c.take<T>(n);
        rb = c.take<T>(n);
        ca = c.take<T>(n);
        cb = c.take<T>(n);
        outdeg = c.take<int32_t>(n);
        flag = c.take<int32_t>(n);
        pos = c.take<int32_t>((size_t)n + 1);
        row_id = c.take<int32_t>(n);
        row_begin = c.take<int32_t>((size_t)n + 1);
        row_deg = c.take<int32_t>(n);
        bare = c.take<int32_t>(n);
        tile = c.take<int32_t>((size_t)tiles + 1);
        head = c.take<double>((size_t)tiles + 1);
        tail = c.take<double>((size_t)tiles + 1);
        bs = c.take<int64_t>(scan_scratch_words(n));
        ps = c.take<double>(nparts);
        pl = c.take<double>(nparts);
        sc = c.take<PrScalars>(1);
        bare_count = c.take<int32_t>(2);
        done = c.take<int32_t>(1);
        hist = c.take<double>(o->iterations > 0 ? o->iterations : 1);
    };
    Carver sizing(nullptr);
    carve(sizing);
    GHB_TRY(ws_reserve(ws, sizing.off));
    Carver c(ws->scratch);
    carve(c);

    const double d = o->damping;
    // One limit for every call: it belongs to the process, and another thread's
    // call on another graph may lie between this and the launches below.
    GHB_CUDA_TRY(cudaFuncSetAttribute(pr_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrMaxSmem));
    // ps, pl, sc, bare_count and done lie behind one another.
    GHB_CUDA_TRY(cudaMemsetAsync(ps, 0, (size_t)(reinterpret_cast<char*>(done + 1) - reinterpret_cast<char*>(ps)), st));
    GHB_TRY(launch(ws, pr_init_kernel<T>, dim3(grid_init), dim3(kPrThreads), 0, n, out_rp, outdeg, ra, ca, cb, ps));
    GHB_TRY(launch(ws, pr_reduce_kernel, dim3(1), dim3(kPrThreads), 0, (const double*)ps, (const double*)pl, nparts, n, d,
                   sc));
    // The non-empty rows, the empty ones, and each tile's first row.
    GHB_TRY(launch(ws, pr_row_flags_kernel, dim3(grid_for(n, 256, g)), dim3(256), 0, n, in_rp, flag));
    GHB_TRY(scan_exclusive_i32(ws, flag, pos, n, bs));
    GHB_TRY(launch(ws, pr_row_lists_kernel, dim3(grid_for(n, 256, g)), dim3(256), 0, n, in_rp, (const int32_t*)pos,
                   (const int32_t*)outdeg, row_id, row_begin, row_deg, bare, bare_count));
    const PrRows rows{row_id, row_begin, row_deg, tile, (int32_t)m, tiles};
    if (tiles)
        GHB_TRY(launch(ws, pr_tile_rows_kernel, dim3(grid_for(tiles, 256, g)), dim3(256), 0, (const int32_t*)(pos + n),
                       (const int32_t*)row_begin, tiles, tile));

    T *r_cur = ra, *r_nxt = rb, *c_cur = ca, *c_nxt = cb;
    const bool track = o->tolerance > 0 || o->l1_history != nullptr;
    int it = 0;
    for (; it < o->iterations; ++it) {
        if (tiles)
            GHB_TRY(launch(ws, pr_tile_kernel<T>, dim3(grid_rows), dim3(pthreads), smem, rows, n, in_col,
                           (const T*)c_cur, (const T*)r_cur, r_nxt, c_nxt, (const PrScalars*)sc,
                           d, track ? 1 : 0, head, tail, ps, pl, cache_elems));
        GHB_TRY(launch(ws, pr_finish_kernel<T>, dim3(grid_fin), dim3(kPrThreads), 0, rows, n, (const int32_t*)bare,
                       (const int32_t*)bare_count, track || it + 1 == o->iterations ? 1 : 0, (const double*)head, (const double*)tail, (const int32_t*)outdeg, (const T*)r_cur, r_nxt, c_nxt,
                       sc, d, track ? 1 : 0, ps, pl, (int)grid_rows, nparts, hist, it, done));
        std::swap(r_cur, r_nxt);
        std::swap(c_cur, c_nxt);
        if (o->tolerance > 0) {
            GHB_CUDA_TRY(cudaMemcpyAsync(ws->host_pinned, sc, sizeof(PrScalars), cudaMemcpyDeviceToHost, st));
            GHB_CUDA_TRY(cudaStreamSynchronize(st));
            const PrScalars* h = reinterpret_cast<const PrScalars*>(ws->host_pinned);
            if (h->l1 <= o->tolerance) {
                ++it;
                break;
            }
        }
    }
    GHB_TRY(launch(ws, pr_to_f64_kernel<T>, dim3(grid_for(n, 256, ws->num_sms * 8)), dim3(256), 0, (const T*)r_cur,
                   perm, rank_out, n));
    if (o->l1_history && it > 0) {
        GHB_CUDA_TRY(cudaMemcpyAsync(o->l1_history, hist, sizeof(double) * it, cudaMemcpyDeviceToHost, st));
        GHB_CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (iters_run) *iters_run = it;
    return GHB_OK;
}

}  // namespace

// Rows in the order of a degree ranking (perm[caller's id]; rank in the
// caller's ids), m entries.
int pagerank_run(ghb_workspace* ws, int32_t n, int64_t m, const int32_t* in_rp, const int32_t* in_col,
                 const int32_t* out_rp, const int32_t* perm, const ghb_pr_options* o, double* rank,
                 int32_t* iters_run) {
    if (o->precision == GHB_PR_FP64)
        return pagerank_impl<double>(ws, n, m, in_rp, in_col, out_rp, o, rank, iters_run, perm);
    return pagerank_impl<float>(ws, n, m, in_rp, in_col, out_rp, o, rank, iters_run, perm);
}

}  // namespace ghb

using namespace ghb;

extern "C" int ghb_pagerank(ghb_workspace* ws, int32_t n, const int32_t* in_rowptr, const int32_t* in_col,
                            const int32_t* out_rowptr, const ghb_pr_options* options, double* rank,
                            int32_t* iterations_run) {
    ws = ws_resolve(ws);
    GHB_REQUIRE(ws, "no workspace");
    GHB_REQUIRE(n >= 1, "n must be >= 1");
    GHB_REQUIRE(in_rowptr && out_rowptr && rank && options, "NULL argument");
    GHB_REQUIRE(options->iterations >= 0, "iterations < 0");
    GHB_REQUIRE(options->precision == GHB_PR_FP64 || options->precision == GHB_PR_FP32_KAHAN,
                "bad precision");
    if (options->precision == GHB_PR_FP64)
        return pagerank_impl<double>(ws, n, -1, in_rowptr, in_col, out_rowptr, options, rank, iterations_run, nullptr);
    return pagerank_impl<float>(ws, n, -1, in_rowptr, in_col, out_rowptr, options, rank, iterations_run, nullptr);
}
