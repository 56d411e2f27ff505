// Resident graph handle: the caller's CSR relabelled by degree on the GPU.
//
// New ids rank vertices by total degree, descending (ties by old id), so
//  * hubs have the smallest ids: sorted rows list them first, a bottom-up BFS
//    step meets a frontier hub on its first probe, and gathers of hub values
//    (PageRank contributions, BFS frontier words) hit a few cache lines;
//  * vertices with no entries form the tail [n_active, n): traversal and
//    label kernels skip it;
//  * "v < u" orients every undirected edge from the lower- to the higher-
//    degree end, so triangle counting reads an oriented row as the prefix of
//    the sorted row that precedes u (no copy).
// The relabelling is a one-time step per graph (like the reference's toCSR,
// GPU_csr.hpp:282-339); results are mapped back to the caller's ids.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "graph.cuh"
#include "scan.cuh"
#include "sorted_rows.cuh"

namespace ghb {
namespace {

__device__ __forceinline__ uint64_t degree_key(uint32_t d, int64_t v) {
    return ((uint64_t)(0xFFFFFFFFu - d) << 32) | (uint64_t)(uint32_t)v;
}

// Degree keys (descending degree, then id).  When rowptr (and the in-CSR's)
// start on 16-byte boundaries a thread takes four vertices with one 16-byte
// load of rowptr[4q..4q+3] plus rowptr[4q+4].
__global__ void degree_key_kernel(int32_t n, const int32_t* __restrict__ out_rp, const int32_t* __restrict__ in_rp,
                                  uint64_t* keys) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const bool vec = ((uintptr_t)out_rp & 15) == 0 && (!in_rp || ((uintptr_t)in_rp & 15) == 0);
    int64_t v0 = 0;
    if (vec) {
        const int64_t quads = n / 4;
        for (int64_t q = tid; q < quads; q += stride) {
            const int4 a = reinterpret_cast<const int4*>(out_rp)[q];
            const int32_t nx = out_rp[4 * q + 4];
            uint32_t d0 = a.y - a.x, d1 = a.z - a.y, d2 = a.w - a.z, d3 = nx - a.w;
            if (in_rp) {
                const int4 b = reinterpret_cast<const int4*>(in_rp)[q];
                const int32_t ny = in_rp[4 * q + 4];
                d0 += b.y - b.x;
                d1 += b.z - b.y;
                d2 += b.w - b.z;
                d3 += ny - b.w;
            }
            keys[4 * q] = degree_key(d0, 4 * q);
            keys[4 * q + 1] = degree_key(d1, 4 * q + 1);
            keys[4 * q + 2] = degree_key(d2, 4 * q + 2);
            keys[4 * q + 3] = degree_key(d3, 4 * q + 3);
        }
        v0 = quads * 4;
    }
    for (int64_t v = v0 + tid; v < n; v += stride) {
        uint32_t d = (uint32_t)(out_rp[v + 1] - out_rp[v]);
        if (in_rp) d += (uint32_t)(in_rp[v + 1] - in_rp[v]);
        keys[v] = degree_key(d, v);
    }
}

__global__ void perm_from_keys_kernel(int32_t n, const uint64_t* __restrict__ keys, int32_t* perm, int32_t* iperm,
                                      int32_t* n_active) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        const int32_t old = (int32_t)(uint32_t)k;
        iperm[i] = old;
        perm[old] = (int32_t)i;
        const bool zero = (uint32_t)(k >> 32) == 0xFFFFFFFFu;
        const bool prev_nonzero = i == 0 || (uint32_t)(keys[i - 1] >> 32) != 0xFFFFFFFFu;
        if (zero && prev_nonzero) *n_active = (int32_t)i;
    }
}

// One key per entry: (new row << bits) | new col, value = entry index.  A warp takes
// 32 rows: those of 32 entries or more one after another, the others packed
// over a scan of their lengths, four columns and their new ids in flight per
// lane either way.  Rows of kRelabelLong entries or more are listed (longer_rows
// [0] their number) for a block each.  Bound by the gathers of the new ids; with
// a warp per row the longest row's chain of loads set the pace (RMAT-22: 1.85 ms;
// 0.60 and 0.35 for the long rows).
constexpr int32_t kRelabelLong = 2048;
__global__ void __launch_bounds__(256) relabel_keys_kernel(int32_t n, const int32_t* __restrict__ rp,
                                                           const int32_t* __restrict__ col,
                                                           const int32_t* __restrict__ perm, int bits, uint64_t* keys,
                                                           uint32_t* vals, int32_t* longer_rows) {
    constexpr int kB = 4;
    const int lane = lane_id();
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    auto emit = [&](const int64_t (&j)[kB], const bool (&ok)[kB], const int32_t (&row)[kB]) {
        int32_t c[kB];
#pragma unroll
        for (int q = 0; q < kB; ++q) c[q] = ok[q] ? col[j[q]] : 0;
#pragma unroll
        for (int q = 0; q < kB; ++q) c[q] = ok[q] ? perm[c[q]] : 0;
#pragma unroll
        for (int q = 0; q < kB; ++q)
            if (ok[q]) {
                keys[j[q]] = ((uint64_t)(uint32_t)row[q] << bits) | (uint64_t)(uint32_t)c[q];
                if (vals) vals[j[q]] = (uint32_t)j[q];
            }
    };
    for (int64_t base = warp * 32; base < n; base += nwarps * 32) {
        const int64_t u = base + lane;
        const int32_t b = u < n ? rp[u] : 0;
        int32_t e = u < n ? rp[u + 1] : 0;
        const int32_t nu = u < n ? perm[u] : 0;
        unsigned longer = __ballot_sync(0xffffffffu, e - b >= 32);
        while (longer) {
            const int l = __ffs(longer) - 1;
            longer &= longer - 1;
            const int32_t lb = __shfl_sync(0xffffffffu, b, l), le = __shfl_sync(0xffffffffu, e, l);
            const int32_t lu = __shfl_sync(0xffffffffu, nu, l);
            if (le - lb >= kRelabelLong) {
                if (lane == 0) longer_rows[1 + atomicAdd(longer_rows, 1)] = (int32_t)(base + l);
                continue;
            }
            for (int64_t j0 = lb; j0 < le; j0 += 32 * kB) {
                int64_t j[kB];
                bool ok[kB];
                int32_t row[kB];
#pragma unroll
                for (int q = 0; q < kB; ++q) {
                    j[q] = j0 + 32 * q + lane;
                    ok[q] = j[q] < le;
                    row[q] = lu;
                }
                emit(j, ok, row);
            }
        }
        if (e - b >= 32) e = b;
        int32_t incl = e - b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        const int32_t excl = incl - (e - b), total = __shfl_sync(0xffffffffu, incl, 31);
        for (int32_t k0 = 0; k0 < total; k0 += 32 * kB) {
            int64_t j[kB];
            bool ok[kB];
            int32_t row[kB];
#pragma unroll
            for (int q = 0; q < kB; ++q) {
                const int32_t k = k0 + 32 * q + lane;
                int owner = 0;
#pragma unroll
                for (int s = 16; s >= 1; s >>= 1) {
                    const int32_t at = __shfl_sync(0xffffffffu, excl, owner + s);
                    if (at <= k) owner += s;
                }
                const int32_t ob = __shfl_sync(0xffffffffu, b, owner), oe = __shfl_sync(0xffffffffu, excl, owner);
                row[q] = __shfl_sync(0xffffffffu, nu, owner);
                ok[q] = k < total;
                j[q] = (int64_t)ob + (k - oe);
            }
            emit(j, ok, row);
        }
    }
}

// The long rows, a block each.
__global__ void __launch_bounds__(1024) relabel_long_kernel(const int32_t* __restrict__ rp,
                                                            const int32_t* __restrict__ col,
                                                            const int32_t* __restrict__ perm, int bits, uint64_t* keys,
                                                            uint32_t* vals, const int32_t* __restrict__ longer_rows) {
    constexpr int kB = 4;
    const int32_t rows = longer_rows[0];
    for (int32_t i = blockIdx.x; i < rows; i += gridDim.x) {
        const int32_t u = longer_rows[1 + i];
        const int64_t b = rp[u], e = rp[u + 1];
        const uint64_t nu = (uint64_t)(uint32_t)perm[u] << bits;
        for (int64_t j0 = b + threadIdx.x; j0 < e; j0 += 1024 * kB) {
            int32_t c[kB];
#pragma unroll
            for (int q = 0; q < kB; ++q) c[q] = j0 + 1024 * q < e ? col[j0 + 1024 * q] : 0;
#pragma unroll
            for (int q = 0; q < kB; ++q) c[q] = j0 + 1024 * q < e ? perm[c[q]] : 0;
#pragma unroll
            for (int q = 0; q < kB; ++q) {
                const int64_t j = j0 + 1024 * q;
                if (j >= e) break;
                keys[j] = nu | (uint64_t)(uint32_t)c[q];
                if (vals) vals[j] = (uint32_t)j;
            }
        }
    }
}

// Columns, weights and row offsets of the sorted keys in one pass over them;
// *repeat is set when a row holds an entry twice.
__global__ void __launch_bounds__(256) relabel_out_kernel(const uint64_t* __restrict__ keys,
                                                          const uint32_t* __restrict__ vals, int64_t m, int32_t n,
                                                          int bits, const double* __restrict__ w, int32_t* col,
                                                          double* w_out, int32_t* __restrict__ rowptr,
                                                          int32_t* repeat) {
    constexpr int kItems = 4;  // weight gathers in flight per thread
    __shared__ RowGaps gaps;
    if (threadIdx.x == 0) gaps.count = 0;
    __syncthreads();
    const uint64_t mask = (1ull << bits) - 1;
    bool twice = false;
    for (int64_t i0 = blockIdx.x * (int64_t)(256 * kItems) + threadIdx.x; i0 <= m;
         i0 += (int64_t)gridDim.x * (256 * kItems)) {
        uint32_t v[kItems];
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const int64_t i = i0 + q * 256;
            v[q] = w_out && i < m ? vals[i] : 0u;
        }
        double x[kItems];
#pragma unroll
        for (int q = 0; q < kItems; ++q) x[q] = w_out && i0 + q * 256 < m ? w[v[q]] : 0.0;
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const int64_t i = i0 + q * 256;
            if (i > m) break;
            const uint64_t k = i < m ? keys[i] : (uint64_t)n << bits;
            const uint64_t kp = i > 0 ? keys[i - 1] : 0;
            const int64_t prev = i > 0 ? (int64_t)(kp >> bits) : -1, cur = (int64_t)(k >> bits);
            if (cur > prev) fill_rows(gaps, rowptr, prev + 1, cur, (int32_t)i);
            if (i < m) {
                col[i] = (int32_t)(k & mask);
                if (w_out) w_out[i] = x[q];
                twice |= i > 0 && k == kp;
            }
        }
    }
    if (twice) *repeat = 1;
    __syncthreads();
    fill_long_rows(gaps, rowptr);
}

__global__ void outdeg_kernel(int32_t n, const int32_t* __restrict__ rp, int32_t* outdeg) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        outdeg[v] = rp[v + 1] - rp[v];
}

template <class T>
__global__ void map_back_kernel(int32_t n, const int32_t* __restrict__ perm, const T* __restrict__ src, T* dst) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        dst[v] = src[perm[v]];
}

int bits_for_n(int32_t n) {
    int bits = 1;
    while (bits < 31 && (1ll << bits) < (int64_t)n) ++bits;
    return bits;
}

}  // namespace

// perm / iperm of the degree ranking (total degree with in_rp, descending, ties
// by id); *n_active (device, preset to n) gets the first id without entries.
int rank_by_degree(ghb_workspace* ws, int32_t n, const int32_t* out_rp, const int32_t* in_rp, int32_t* perm,
                   int32_t* iperm, int32_t** n_active) {
    // Ids enter in order and the sort is stable: only the degrees are sorted.
    size_t sort_tmp = 0;
    {
        cub::DoubleBuffer<uint64_t> dk(nullptr, nullptr);
        cub::DeviceRadixSort::SortKeys(nullptr, sort_tmp, dk, (int64_t)n, 32, 64);
    }
    uint64_t *k0, *k1;
    void* tmp;
    int32_t* nact;
    auto carve = [&](Carver& c) {
        k0 = c.take<uint64_t>(n);
        k1 = c.take<uint64_t>(n);
        nact = c.take<int32_t>(8);
        tmp = c.take<char>(sort_tmp);
    };
    Carver sizing(nullptr);
    carve(sizing);
    GHB_TRY(ws_reserve(ws, sizing.off));
    Carver c(ws->scratch);
    carve(c);
    const unsigned gr = grid_for(n, 256, ws->num_sms * 8);
    GHB_TRY(launch(ws, degree_key_kernel, dim3(gr), dim3(256), 0, n, out_rp, in_rp, k0));
    cub::DoubleBuffer<uint64_t> dk(k0, k1);
    size_t tb = sort_tmp;
    GHB_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp, tb, dk, (int64_t)n, 32, 64, ws->stream));
    ws->launches++;
    const int32_t nn = n;
    GHB_CUDA_TRY(cudaMemcpyAsync(nact, &nn, sizeof(int32_t), cudaMemcpyHostToDevice, ws->stream));
    GHB_TRY(launch(ws, perm_from_keys_kernel, dim3(gr), dim3(256), 0, n, (const uint64_t*)dk.Current(), perm, iperm, nact));
    *n_active = nact;
    return GHB_OK;
}

// Relabel one CSR (rows and columns through perm), rows sorted, weights
// carried along; *repeat (device) is set when a row holds an entry twice.
int relabel_csr(ghb_workspace* ws, int32_t n, int64_t m, const int32_t* rp, const int32_t* col, const double* w,
                const int32_t* perm, int32_t* rp_out, int32_t* col_out, double* w_out, int32_t* repeat) {
    if (m == 0) {
        GHB_CUDA_TRY(cudaMemsetAsync(rp_out, 0, sizeof(int32_t) * ((size_t)n + 1), ws->stream));
        return GHB_OK;
    }
    const int bits = bits_for_n(n);
    const bool want_vals = w != nullptr && w_out != nullptr;
    size_t sort_tmp = 0;
    {
        cub::DoubleBuffer<uint64_t> dk(nullptr, nullptr);
        cub::DoubleBuffer<uint32_t> dv(nullptr, nullptr);
        if (want_vals) cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, dk, dv, m, 0, 2 * bits);
        else cub::DeviceRadixSort::SortKeys(nullptr, sort_tmp, dk, m, 0, 2 * bits);
    }
    auto carve = [&](Carver& c, uint64_t** k0, uint64_t** k1, uint32_t** v0, uint32_t** v1, void** tmp) {
        *k0 = c.take<uint64_t>(m);
        *k1 = c.take<uint64_t>(m);
        *v0 = want_vals ? c.take<uint32_t>(m) : nullptr;
        *v1 = want_vals ? c.take<uint32_t>(m) : nullptr;
        *tmp = c.take<char>(sort_tmp);
    };
    uint64_t *k0, *k1;
    uint32_t *v0, *v1;
    void* tmp;
    Carver sizing(nullptr);
    carve(sizing, &k0, &k1, &v0, &v1, &tmp);
    GHB_TRY(ws_reserve(ws, sizing.off));
    Carver c(ws->scratch);
    carve(c, &k0, &k1, &v0, &v1, &tmp);
    const unsigned g = ws->num_sms * 8;
    // The list of long rows (fewer than m / kRelabelLong + 1) lies where the sort
    // writes later.
    int32_t* longer_rows = reinterpret_cast<int32_t*>(k1);
    GHB_CUDA_TRY(cudaMemsetAsync(longer_rows, 0, sizeof(int32_t), ws->stream));
    GHB_TRY(launch(ws, relabel_keys_kernel, dim3(grid_for(n, 256, g)), dim3(256), 0, n, rp, col, perm, bits, k0, v0,
                   longer_rows));
    if (m >= kRelabelLong)
        GHB_TRY(launch(ws, relabel_long_kernel, dim3(ws->num_sms * 2), dim3(1024), 0, rp, col, perm, bits, k0, v0,
                       (const int32_t*)longer_rows));
    cub::DoubleBuffer<uint64_t> dk(k0, k1);
    cub::DoubleBuffer<uint32_t> dv(v0, v1);
    size_t tb = sort_tmp;
    if (want_vals) GHB_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, dk, dv, m, 0, 2 * bits, ws->stream));
    else GHB_CUDA_TRY(cub::DeviceRadixSort::SortKeys(tmp, tb, dk, m, 0, 2 * bits, ws->stream));
    ws->launches++;
    return launch(ws, relabel_out_kernel, dim3(grid_for(m + 1, 256 * 4, g)), dim3(256), 0, (const uint64_t*)dk.Current(),
                  (const uint32_t*)(want_vals ? dv.Current() : nullptr), m, n, bits, w, col_out,
                  want_vals ? w_out : (double*)nullptr, rp_out, repeat);
}

int map_back_i32(ghb_workspace* ws, const ghb_graph* g, const int32_t* src_new, int32_t* dst_old) {
    return launch(ws, map_back_kernel<int32_t>, dim3(grid_for(g->n, 256, ws->num_sms * 8)), dim3(256), 0, g->n,
                  (const int32_t*)g->perm, src_new, dst_old);
}
int map_source(ghb_workspace* ws, const ghb_graph* g, int32_t src, int32_t* src_new) {
    int32_t* hp = reinterpret_cast<int32_t*>(ws->host_pinned);
    GHB_CUDA_TRY(cudaMemcpyAsync(hp, g->perm + src, sizeof(int32_t), cudaMemcpyDeviceToHost, ws->stream));
    GHB_CUDA_TRY(cudaStreamSynchronize(ws->stream));
    *src_new = hp[0];
    return GHB_OK;
}

int map_back_f64(ghb_workspace* ws, const ghb_graph* g, const double* src_new, double* dst_old) {
    return launch(ws, map_back_kernel<double>, dim3(grid_for(g->n, 256, ws->num_sms * 8)), dim3(256), 0, g->n,
                  (const int32_t*)g->perm, src_new, dst_old);
}
int map_back_i64(ghb_workspace* ws, const ghb_graph* g, const int64_t* src_new, int64_t* dst_old) {
    return launch(ws, map_back_kernel<int64_t>, dim3(grid_for(g->n, 256, ws->num_sms * 8)), dim3(256), 0, g->n,
                  (const int32_t*)g->perm, src_new, dst_old);
}

}  // namespace ghb

using namespace ghb;

extern "C" {

int ghb_graph_destroy(ghb_graph* g) {
    if (!g) return GHB_OK;
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(g->device);
    cudaFree(g->slab);
    cudaFree(g->sw_col);
    cudaFree(g->sw_w);
    cudaFree(g->sw_le);
    cudaSetDevice(cur);
    delete g;
    return GHB_OK;
}

int ghb_graph_create(ghb_workspace* ws, int32_t n, const int32_t* out_rowptr, const int32_t* out_col,
                     const double* out_w, const int32_t* in_rowptr, const int32_t* in_col, const double* in_w,
                     ghb_graph** out) {
    ws = ws_resolve(ws);
    GHB_REQUIRE(ws, "no workspace");
    GHB_REQUIRE(out, "NULL out");
    GHB_REQUIRE(n >= 1, "n must be >= 1");
    GHB_REQUIRE(out_rowptr, "NULL out_rowptr");
    *out = nullptr;
    cudaStream_t st = ws->stream;
    const bool directed = in_rowptr != nullptr && in_rowptr != out_rowptr;
    int32_t* hp = reinterpret_cast<int32_t*>(ws->host_pinned);
    GHB_CUDA_TRY(cudaMemcpyAsync(hp, out_rowptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    if (directed) GHB_CUDA_TRY(cudaMemcpyAsync(hp + 1, in_rowptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    GHB_CUDA_TRY(cudaStreamSynchronize(st));
    ghb_graph* g = new ghb_graph();
    g->n = n;
    g->m = hp[0];
    g->m_in = directed ? hp[1] : hp[0];
    g->directed = directed;
    g->weighted = out_w != nullptr;
    GHB_CUDA_TRY(cudaGetDevice(&g->device));
    GHB_CUDA_TRY(cudaEventRecord(ws->ev_a, st));
    auto fail = [&](int s) {
        ghb_graph_destroy(g);
        return s;
    };
    int s = GHB_OK;
#define GG_TRY(x)                 \
    do {                          \
        s = (x);                  \
        if (s != GHB_OK) return fail(s); \
    } while (0)
    // One allocation for all of the handle's arrays (an allocation and its
    // release each cost hundreds of microseconds at these sizes).
    auto carve = [&](Carver& c) {
        g->perm = c.take<int32_t>(n);
        g->iperm = c.take<int32_t>(n);
        g->rowptr = c.take<int32_t>((size_t)n + 1);
        g->col = c.take<int32_t>(std::max<int64_t>(g->m, 1));
        if (g->weighted) g->w = c.take<double>(std::max<int64_t>(g->m, 1));
        g->outdeg = c.take<int32_t>(n);
        if (directed) {
            g->in_rowptr = c.take<int32_t>((size_t)n + 1);
            g->in_col = c.take<int32_t>(std::max<int64_t>(g->m_in, 1));
            if (in_w) g->in_w = c.take<double>(std::max<int64_t>(g->m_in, 1));
            g->all_rowptr = c.take<int32_t>((size_t)n + 1);
            g->all_col = c.take<int32_t>(std::max<int64_t>(g->m + g->m_in, 1));
        }
    };
    Carver need(nullptr);
    carve(need);
    {
        const cudaError_t e = cudaMalloc(&g->slab, need.off);
        if (e != cudaSuccess) {
            set_error(std::string("resident graph: ") + cudaGetErrorString(e));
            g->slab = nullptr;
            return fail(e == cudaErrorMemoryAllocation ? GHB_ERR_OUT_OF_MEMORY : GHB_ERR_CUDA);
        }
    }
    g->device_bytes = (int64_t)need.off;
    Carver slab(g->slab);
    carve(slab);
    if (!directed) {
        g->in_rowptr = g->rowptr;
        g->in_col = g->col;
        g->in_w = g->w;
        g->all_rowptr = g->rowptr;
        g->all_col = g->col;
    }
    // 1. degree ranking -> perm / iperm / n_active
    {
        int32_t* nact = nullptr;
        GG_TRY(rank_by_degree(ws, n, out_rowptr, directed ? in_rowptr : (const int32_t*)nullptr, g->perm, g->iperm, &nact));
        cudaError_t e = cudaMemcpyAsync(hp, nact, sizeof(int32_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return fail(GHB_ERR_CUDA);
        g->n_active = hp[0];
    }
    // 2. relabelled CSRs
    int32_t* repeat = reinterpret_cast<int32_t*>(ws->dev_small);  // [0] out-rows, [1] in-rows (not used)
    GG_TRY(cudaMemsetAsync(repeat, 0, 2 * sizeof(int32_t), st) == cudaSuccess ? GHB_OK : GHB_ERR_CUDA);
    GG_TRY(relabel_csr(ws, n, g->m, out_rowptr, out_col, out_w, g->perm, g->rowptr, g->col, g->w, repeat));
    if (directed)
        GG_TRY(relabel_csr(ws, n, g->m_in, in_rowptr, in_col, in_w, g->perm, g->in_rowptr, g->in_col, g->in_w,
                           repeat + 1));
    GG_TRY(launch(ws, outdeg_kernel, dim3(grid_for(n, 256, ws->num_sms * 8)), dim3(256), 0, n,
                  (const int32_t*)g->rowptr, g->outdeg));
    if (directed)
        GG_TRY(ghb_csr_merge_in_out(ws, n, g->in_rowptr, g->in_col, g->rowptr, g->col, g->all_rowptr, g->all_col));
    GG_TRY(cudaMemcpyAsync(hp + 2, repeat, sizeof(int32_t), cudaMemcpyDeviceToHost, st) == cudaSuccess ? GHB_OK
                                                                                                     : GHB_ERR_CUDA);
#undef GG_TRY
    GHB_CUDA_TRY(cudaEventRecord(ws->ev_b, st));
    GHB_CUDA_TRY(cudaEventSynchronize(ws->ev_b));
    g->repeats = hp[2] != 0;
    cudaEventElapsedTime(&g->build_ms, ws->ev_a, ws->ev_b);
    *out = g;
    return GHB_OK;
}

int ghb_graph_info(const ghb_graph* g, int64_t* m, int32_t* n_active, int64_t* device_bytes, float* build_ms) {
    GHB_REQUIRE(g, "NULL graph");
    if (m) *m = g->m;
    if (n_active) *n_active = g->n_active;
    if (device_bytes) *device_bytes = g->device_bytes;
    if (build_ms) *build_ms = g->build_ms;
    return GHB_OK;
}

int ghb_graph_perm(const ghb_graph* g, const int32_t** perm, const int32_t** iperm) {
    GHB_REQUIRE(g, "NULL graph");
    if (perm) *perm = g->perm;
    if (iperm) *iperm = g->iperm;
    return GHB_OK;
}

}  // extern "C"
