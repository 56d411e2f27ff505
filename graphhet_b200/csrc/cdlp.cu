// Community detection by synchronous label propagation (replaces
// GPU_CDLP_csr.cuh:28-210, which gathers every row's labels into an E-length
// array and segment-sorts all E keys each iteration).  Semantics of the CPU
// path (CPU_Community_Detection.hpp:12-64): the new label of v is the most
// frequent label among its row's entries, the smallest such label on ties; a
// vertex with an empty row keeps its label.  Labels start as vertex ids.
//
// Rows are classed by length once per call and each class has its own
// kernel, so no row pays for another's size:
//   0        keep the label
//   1..32    W lanes per row (W = 2..32): bitonic sort of the W labels in
//            registers through shuffles, run lengths by ballot
//   33..256  one warp per row, its labels in registers; open-addressing
//            (label -> count) table of up to 512 slots in shared memory
//   257..1024 one block per row, 2048-slot shared-memory table (16 KB, so
//            eight blocks fit an SM)
//   1025..2048 one block per row, 4096-slot shared-memory table (32 KB)
//   2049..4096 one block per row, 8192-slot shared-memory table
//   > 4096   the row is cut into chunks of 2048 entries, each a block: the
//            chunk counts its labels in a shared-memory table, then adds each
//            distinct (label, count) to the row's table in global scratch and
//            lists the slots it claimed; the last chunk of a row to finish
//            writes its label, and a write-only pass empties the claimed
//            slots.  No row waits on one block, and once labels converge a
//            chunk sends a few global atomics, not 2048.
// From class 6 on, a row is first tried for a label that holds more than half
// of it (the leading label of 32 of its entries, counted in full): once
// communities have formed nearly every row has one, and such a row costs its
// label gathers and no table.
// Every insert returns the key (count after it, -label); a label's last insert
// sees its final count, so the max-reduction of those keys yields the most
// frequent label with the smallest-label tie-break, and no table is scanned
// for it.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace ghb {
namespace {

// 0:empty 1..5: W=2,4,8,16,32  6:warp 7:block (2048 slots) 8:block (4096 slots)
// 9:block (8192 slots) 10:chunked
constexpr int kCdlpClasses = 11;
constexpr int kSumLongSlot = 15;  // counts[15]: entries of the chunked-class rows
constexpr int kSumSlot = 14;      // counts[14]: of all rows
constexpr int32_t kEmpty = -1;
constexpr int32_t kWarpSlots = 512;
constexpr int32_t kSmallBlockSlots = 2048;
constexpr int32_t kMidBlockSlots = 4096;
constexpr int32_t kBlockSlots = 8192;
constexpr int32_t kLongRow = kBlockSlots / 2;  // longer rows are chunked
constexpr int32_t kChunk = 2048;               // entries per chunk of a chunked-class row
constexpr int32_t kChunkSlots = 2 * kChunk;    // its shared-memory table (32 KB)
constexpr int kCdlpThreads = 256;
constexpr int32_t kCheckRows = 1 << 17;  // vertices from which an iteration is split by what its rows need

__device__ __forceinline__ int cdlp_class(int32_t d) {
    if (d == 0) return 0;
    if (d <= 2) return 1;
    if (d <= 4) return 2;
    if (d <= 8) return 3;
    if (d <= 16) return 4;
    if (d <= 32) return 5;
    if (d <= 256) return 6;
    if (d <= 1024) return 7;
    if (d <= 2048) return 8;
    if (d <= kLongRow) return 9;
    return 10;
}

// Slots of a chunked-class row's global table: the power of two >= 2 d.
__host__ __device__ __forceinline__ uint32_t global_cap(int32_t d) {
    uint32_t c = 1;
    while (c < 2u * (uint32_t)d) c <<= 1;
    return c;
}

__device__ __forceinline__ uint32_t hash_label(int32_t x) {
    uint32_t h = (uint32_t)x * 0x9E3779B1u;
    return h ^ (h >> 16);
}

// Packs (count, label) so that a larger key = more frequent, then smaller label.
__device__ __forceinline__ unsigned long long pack_best(uint32_t count, int32_t label) {
    return ((unsigned long long)count << 32) | (unsigned long long)(0x7FFFFFFFu - (uint32_t)label);
}
__device__ __forceinline__ int32_t unpack_label(unsigned long long k) {
    return (int32_t)(0x7FFFFFFFu - (uint32_t)(k & 0xFFFFFFFFull));
}

// Adds `count` to label x in an open-addressing table of `slots` (power of two)
// entries, K = labels, C = counts, and returns the key (count after this
// add, label).  A label's count only grows and its last insert sees the
// final count, so the largest key returned over a row names its most frequent
// label (smallest on ties) without a scan of the table.
__device__ __forceinline__ unsigned long long table_add(int32_t* K, int32_t* C, uint32_t slots, int32_t x,
                                                        int32_t count) {
    uint32_t h = hash_label(x) & (slots - 1);
    while (true) {
        const int32_t k = atomicCAS(&K[h], kEmpty, x);
        if (k == kEmpty || k == x) return pack_best((uint32_t)(atomicAdd(&C[h], count) + count), x);
        h = (h + 1) & (slots - 1);
    }
}

// The row entries b + r * stride + t (r < R) below e, in registers (-1 past
// e), all loads issued together; rounds that begin past e are skipped by the
// whole warp.  Offsets are below 2^31, so unsigned sums do not wrap.  The
// columns stream past L1, which keeps the labels.
template <int R>
__device__ __forceinline__ void load_cols(int32_t (&x)[R], const int32_t* __restrict__ col, int32_t b, int32_t e,
                                          int stride, int t) {
    const uint64_t pol = policy_evict_first();
    const uint32_t first = (uint32_t)b + (uint32_t)(t & ~31), lane = (uint32_t)t & 31u;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t j0 = first + (uint32_t)(r * stride);
        x[r] = -1;
        if (j0 < (uint32_t)e && j0 + lane < (uint32_t)e) x[r] = ld_stream(col + (j0 + lane), pol);
    }
}
// Their labels (never negative), in place.
template <int R>
__device__ __forceinline__ void gather_labels(int32_t (&x)[R], const int32_t* __restrict__ lab) {
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (x[r] >= 0) x[r] = lab[x[r]];
}

// Vertices whose label the last iteration changed, one bit each.  A row
// without one among its entries keeps its label: the same labels give the
// same winner.  Once communities have formed few labels move, and such a row
// costs its columns and bits (n / 8 bytes, mostly in L1) instead of a label
// sector of L2 per entry.  on(): whether the test pays this iteration, by the
// number of changed vertices.
struct CdlpChanged {
    const uint32_t* bits;   // nullptr: not kept (small inputs, first iteration)
    const int32_t* count;
    int32_t limit;
    __device__ __forceinline__ bool on() const { return bits && *count <= limit; }
    __device__ __forceinline__ bool test(int32_t u) const { return u >= 0 && ((bits[u >> 5] >> (u & 31)) & 1u); }
    template <int R>
    __device__ __forceinline__ bool any(const int32_t (&x)[R]) const {
        bool c = false;
#pragma unroll
        for (int r = 0; r < R; ++r) c |= test(x[r]);
        return c;
    }
};

// The bits and their number from an iteration's labels before and after; one
// atomic a block on the number (with one a warp their line set the pace: 8.1 us for
// 490,000 vertices).
__global__ void __launch_bounds__(kCdlpThreads) cdlp_changed_kernel(int32_t n, const int32_t* __restrict__ before,
                                                                    const int32_t* __restrict__ after, uint32_t* bits,
                                                                    int32_t* count) {
    __shared__ int32_t s_count;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    int32_t c = 0;
    for (int64_t v0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll; v0 < n;
         v0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = v0 + lane_id();
        const unsigned m = __ballot_sync(0xffffffffu, v < n && before[v] != after[v]);
        if (lane_id() == 0) bits[v0 >> 5] = m;
        c += __popc(m);
    }
    if (lane_id() == 0 && c) atomicAdd(&s_count, c);
    __syncthreads();
    if (threadIdx.x == 0 && s_count) atomicAdd(count, s_count);
}

// The most frequent label among a full warp's x: the row's likely winner.
// Where it holds more than half of the row it is the answer, whatever the
// rest holds; otherwise it is counted apart, so that the table's atomics do
// not queue on the row's hottest label.
__device__ __forceinline__ int32_t leading_label(int32_t x) {
    const unsigned same = __match_any_sync(0xffffffffu, x);
    const unsigned best = __reduce_max_sync(0xffffffffu, ((unsigned)__popc(same) << 5) | (unsigned)lane_id());
    return __shfl_sync(0xffffffffu, x, (int)(best & 31u));
}

// How many of the warp's labels equal `lead`.
template <int R>
__device__ __forceinline__ int32_t count_label(const int32_t (&x)[R], int32_t lead) {
    int32_t c = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) c += x[r] == lead ? 1 : 0;
    return __reduce_add_sync(0xffffffffu, c);
}

// Inserts the thread's labels other than `lead`; the largest key.
template <int R>
__device__ __forceinline__ unsigned long long insert_labels(int32_t* K, int32_t* C, uint32_t slots,
                                                            const int32_t (&x)[R], int32_t lead) {
    unsigned long long best = 0;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (x[r] >= 0 && x[r] != lead) {
            const unsigned long long key = table_add(K, C, slots, x[r], 1);
            best = key > best ? key : best;
        }
    return best;
}

// The classes' sizes, by blocks: with an atomic on the counters' line for every
// class of every warp, counting took 90 us and filling 93 on RMAT-22; 12 and 22.
__global__ void __launch_bounds__(kCdlpThreads) cdlp_count_classes_kernel(int32_t n, const int32_t* __restrict__ rp,
                                                                          int32_t* counts) {
    __shared__ int32_t s_n[16];
    if (threadIdx.x < 16) s_n[threadIdx.x] = 0;
    __syncthreads();
    int32_t sum = 0;
    for (int64_t v0 = blockIdx.x * (int64_t)kCdlpThreads; v0 < n; v0 += (int64_t)gridDim.x * kCdlpThreads) {
        const int64_t v = v0 + threadIdx.x;
        const int32_t d = v < n ? rp[v + 1] - rp[v] : 0;
        sum += d;
        const int c = v < n ? cdlp_class(d) : -1;
        const unsigned same = __match_any_sync(0xffffffffu, c);
        if (c >= 0 && lane_id() == __ffs(same) - 1) atomicAdd(&s_n[c], __popc(same));
        if (c == 10) atomicAdd(&s_n[kSumLongSlot], d);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane_id() == 0) atomicAdd(&s_n[kSumSlot], sum);
    __syncthreads();
    if (threadIdx.x < 16 && s_n[threadIdx.x]) atomicAdd(counts + threadIdx.x, s_n[threadIdx.x]);
}

// Class lists hold each row as {v, begin, end, 0}: a row kernel reads its
// row's bounds with the row itself, one load instead of two dependent ones.  A
// block places kFillRows x kCdlpThreads rows behind one atomic per class.
constexpr int kFillRows = 4;
__global__ void __launch_bounds__(kCdlpThreads) cdlp_fill_classes_kernel(int32_t n, const int32_t* __restrict__ rp,
                                                                         int32_t* cursor, int4* rows) {
    __shared__ int32_t s_n[kCdlpClasses], s_at[kCdlpClasses];
    const int lane = lane_id();
    constexpr int64_t kTile = kFillRows * kCdlpThreads;
    for (int64_t v0 = blockIdx.x * kTile; v0 < n; v0 += gridDim.x * kTile) {
        if (threadIdx.x < kCdlpClasses) s_n[threadIdx.x] = 0;
        __syncthreads();
        int32_t b[kFillRows], e[kFillRows], at[kFillRows];
        int c[kFillRows];
#pragma unroll
        for (int q = 0; q < kFillRows; ++q) {
            const int64_t v = v0 + q * kCdlpThreads + threadIdx.x;
            b[q] = v < n ? rp[v] : 0;
            e[q] = v < n ? rp[v + 1] : 0;
            c[q] = v < n ? cdlp_class(e[q] - b[q]) : -1;
        }
#pragma unroll
        for (int q = 0; q < kFillRows; ++q) {
            const unsigned same = __match_any_sync(0xffffffffu, c[q]);
            const int leader = __ffs(same) - 1;
            int32_t base = 0;
            if (c[q] >= 0 && lane == leader) base = atomicAdd(&s_n[c[q]], __popc(same));
            at[q] = __shfl_sync(0xffffffffu, base, leader) + __popc(same & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (threadIdx.x < kCdlpClasses && s_n[threadIdx.x])
            s_at[threadIdx.x] = atomicAdd(cursor + threadIdx.x, s_n[threadIdx.x]);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kFillRows; ++q)
            if (c[q] >= 0)
                rows[s_at[c[q]] + at[q]] = make_int4((int32_t)(v0 + q * kCdlpThreads + threadIdx.x), b[q], e[q], 0);
    }
}

__global__ void cdlp_iota_kernel(int32_t* p, int32_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        p[i] = (int32_t)i;
}

// Rows without entries keep their labels.
__device__ __forceinline__ void cdlp_copy_rows(const int4* __restrict__ rows, int32_t count,
                                               const int32_t* __restrict__ lab, int32_t* __restrict__ out, int block,
                                               int nblocks) {
    for (int64_t i = block * (int64_t)kCdlpThreads + threadIdx.x; i < count; i += (int64_t)nblocks * kCdlpThreads) {
        const int32_t v = rows[i].x;
        out[v] = lab[v];
    }
}

// W lanes per row, rows of 1..W entries.  kMin: every label of a row is
// distinct (first iteration), so the row's smallest label is taken directly.
template <int W, bool kMin>
__device__ __forceinline__ void cdlp_small_rows(const int4* __restrict__ rows, int32_t count,
                                                const int32_t* __restrict__ col, const int32_t* __restrict__ lab,
                                                int32_t* __restrict__ out, const CdlpChanged& chg, int block,
                                                int nblocks) {
    const bool check = !kMin && chg.on();
    const int lane = lane_id();
    const int li = lane & (W - 1);
    const int64_t group = (block * (int64_t)kCdlpThreads + threadIdx.x) / W;
    const int64_t ngroups = ((int64_t)nblocks * kCdlpThreads) / W;
    const int64_t rounds = ((int64_t)count + ngroups - 1) / ngroups;
    const unsigned gmask = (W == 32) ? 0xffffffffu : (((1u << W) - 1u) << (lane & ~(W - 1)));
    // The next row's bounds and column load while this row's labels arrive.
    auto row_at = [&](int64_t i) { return i < count ? rows[i] : make_int4(-1, 0, 0, 0); };
    auto col_at = [&](const int4& q) { return li < q.z - q.y ? col[q.y + li] : -1; };
    int4 ri = row_at(group);
    int4 next = row_at(group + ngroups);
    int32_t u = col_at(ri);
    for (int64_t r = 0; r < rounds; ++r) {
        const int64_t i = group + r * ngroups;
        const int32_t v = ri.x, d = ri.z - ri.y, uc = u;
        ri = next;
        u = col_at(next);
        next = row_at(i + 2 * ngroups);
        int32_t x = 0x7FFFFFFF;
        if (check && !__any_sync(0xffffffffu, chg.test(uc))) {  // no row of the warp
            if (li == 0 && i < count) out[v] = lab[v];
            continue;
        }
        if (uc >= 0) x = lab[uc];
        if constexpr (kMin) {
#pragma unroll
            for (int o = W / 2; o > 0; o >>= 1) x = min(x, __shfl_xor_sync(0xffffffffu, x, o));
            if (li == 0 && i < count) out[v] = x;
        } else {
            // Bitonic sort, ascending, within each W-lane group.
#pragma unroll
            for (int k = 2; k <= W; k <<= 1) {
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const int32_t y = __shfl_xor_sync(0xffffffffu, x, j);
                    const bool up = (li & k) == 0;
                    const bool lower = (li & j) == 0;
                    x = (lower == up) ? min(x, y) : max(x, y);
                }
            }
            // Run starts inside the group, then run length = next start - start.
            const int32_t prev = __shfl_up_sync(0xffffffffu, x, 1);
            const bool valid = li < d;
            const bool start = valid && (li == 0 || prev != x);
            const unsigned starts = __ballot_sync(0xffffffffu, start) & gmask;
            unsigned long long best = 0;
            if (start) {
                const unsigned above = starts & ~((2u << lane) - 1u);
                const int next_li = above ? ((__ffs(above) - 1) & (W - 1)) : d;
                best = pack_best((uint32_t)(next_li - li), x);
            }
#pragma unroll
            for (int o = W / 2; o > 0; o >>= 1) {
                const unsigned long long y = __shfl_xor_sync(0xffffffffu, best, o);
                best = y > best ? y : best;
            }
            if (li == 0 && i < count) out[v] = unpack_label(best);
        }
    }
}

// One warp per row of 33..256 entries, all its labels in registers, a table
// of up to kWarpSlots slots per warp in shared memory for the rows that no
// label leads (kMin: the row's smallest label).
template <bool kMin>
__device__ __forceinline__ int32_t cdlp_warp_rows(const int4* __restrict__ rows, int32_t count,
                                               const int32_t* __restrict__ col, const int32_t* __restrict__ lab,
                                               int32_t* __restrict__ out, const CdlpChanged& chg, int block,
                                               int nblocks, int32_t* K, int32_t* C) {
    const bool check = !kMin && chg.on();
    const int lane = lane_id();
    const int64_t warp = (block * (int64_t)kCdlpThreads + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)nblocks * kCdlpThreads) >> 5;
    int32_t tables = 0;  // rows that needed one
    for (int64_t i = warp; i < count; i += nwarps) {
        const int4 ri = rows[i];
        const int32_t v = ri.x, b = ri.y, e = ri.z;
        int32_t x[8];
        load_cols(x, col, b, e, 32, lane);
        if (check && !__any_sync(0xffffffffu, chg.any(x))) {
            if (lane == 0) out[v] = lab[v];
            continue;
        }
        gather_labels(x, lab);
        if (kMin) {
            unsigned m = 0xffffffffu;
#pragma unroll
            for (int r = 0; r < 8; ++r) m = min(m, (unsigned)x[r]);
            m = __reduce_min_sync(0xffffffffu, m);
            if (lane == 0) out[v] = (int32_t)m;
            continue;
        }
        const int32_t lead = leading_label(x[0]);
        const int32_t held = count_label(x, lead);
        if (2 * held > e - b) {
            if (lane == 0) out[v] = lead;
            continue;
        }
        ++tables;
        // Table of the power of two >= 2 x the row (128..512 slots): clearing
        // it costs no more than the row's own inserts.
        uint32_t cap = 64;
        while (cap < 2u * (uint32_t)(e - b)) cap <<= 1;
        for (uint32_t s = lane; s < cap; s += 32) {
            K[s] = kEmpty;
            C[s] = 0;
        }
        __syncwarp();
        unsigned long long best = warp_max(insert_labels(K, C, cap, x, lead));
        const unsigned long long key = pack_best((uint32_t)held, lead);
        if (lane == 0) out[v] = unpack_label(best > key ? best : key);
        __syncwarp();
    }
    return tables;
}

// One warp per row of classes 6 to 9 without a table: rows whose entries did
// not change, or that one label leads, are done; the others go to todo for
// the kernels below.
__device__ __forceinline__ void cdlp_try_rows(const int4* __restrict__ rows, int32_t count,
                                              const int32_t* __restrict__ col, const int32_t* __restrict__ lab,
                                              int32_t* __restrict__ out, const CdlpChanged& chg, int block,
                                              int nblocks, int4* todo, int32_t* ntodo) {
    const bool check = chg.on();
    const int lane = lane_id();
    const int64_t warp = (block * (int64_t)kCdlpThreads + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)nblocks * kCdlpThreads) >> 5;
    int4 ahead = warp < count ? rows[warp] : make_int4(0, 0, 0, 0);
    for (int64_t i = warp; i < count; i += nwarps) {
        const int4 ri = ahead;
        if (i + nwarps < count) ahead = rows[i + nwarps];
        const int32_t b = ri.y, e = ri.z;
        int32_t x[8];
        if (check) {
            bool any = false;
            load_cols(x, col, b, e, 32, lane);
            for (int32_t j = b;;) {
                int32_t y[8];  // the next step's columns, in flight under this one's bits
                const bool more = e - j > 256;
                if (more) load_cols(y, col, j + 256, e, 32, lane);
                any = __any_sync(0xffffffffu, chg.any(x));
                if (any || !more) break;
                j += 256;
#pragma unroll
                for (int r = 0; r < 8; ++r) x[r] = y[r];
            }
            if (!any) {
                if (lane == 0) out[ri.x] = lab[ri.x];
                continue;
            }
        }
        const int32_t lead = leading_label(lab[col[b + lane]]);  // over 32 entries
        int32_t held = 0;
        for (int32_t j = b;; j += 256) {
            load_cols(x, col, j, e, 32, lane);
            gather_labels(x, lab);
#pragma unroll
            for (int r = 0; r < 8; ++r) held += x[r] == lead ? 1 : 0;
            if (e - j <= 256) break;
        }
        held = __reduce_add_sync(0xffffffffu, held);
        if (lane != 0) continue;
        if (2 * held > e - b) out[ri.x] = lead;
        else todo[atomicAdd(ntodo, 1)] = ri;
    }
}

// Classes 0..9 in one launch, each with its own range of blocks
// [first[c], first[c + 1]): an iteration of a small graph is bound by its
// launches, and on a large one a class's last blocks overlap the next.
// kModeMin: the first iteration over distinct labels (classes 0..6).
// kModeTables: class 6 with its tables (classes 0..6).  kModeSmall: classes
// 0..5 alone, whose few registers let a multiprocessor hold its 64 warps (a
// uniform graph of 2^20 vertices of degree 22: 250 us an iteration together
// with the next, 200 apart).  kModeTry: classes 6..9 without tables, which take the L1 that labels and bits are served from; a class of which
// more than one row in kTryShare needed its table last time is left whole to
// the kernels with tables (a row is read twice otherwise).  RMAT-22, ten
// iterations: 13.0 ms with a table for every row, 9.1 with led rows done in the
// table kernels, 7.4 with this pass (an iteration that few labels move in takes
// 0.32 ms where it took 1.3).
enum CdlpMode { kModeMin = 0, kModeTables = 1, kModeTry = 2, kModeSmall = 3 };
constexpr int32_t kTryShare = 8;
struct CdlpLight {
    int32_t off[11];    // rows of class c: [off[c], off[c + 1])
    int32_t first[11];  // blocks of the k-th class from above: class 9 - k, the longest rows first
    int4* todo;         // rows of classes 6..9 that need a table, class c's from off[c] - off[6]
    const int32_t* before;  // how many, by class: last iteration
    int32_t* now;           // this one
};
__device__ __forceinline__ bool needs_tables(int32_t before, int32_t count) {
    return before > count / kTryShare;
}
template <int kMode>
__global__ void __launch_bounds__(kCdlpThreads, kMode == kModeSmall ? 8 : 5)
    cdlp_light_kernel(const int4* __restrict__ rows, CdlpLight q, const int32_t* __restrict__ col,
                      const int32_t* __restrict__ lab, int32_t* __restrict__ out, CdlpChanged chg) {
    constexpr bool M = kMode == kModeMin;
    // The block's class, by selects: indexing the plan would copy it to the
    // stack of every thread.
    int c = 9;
    int32_t f0 = q.first[0], f1 = q.first[1], o0 = q.off[9], o1 = q.off[10];
#pragma unroll
    for (int k = 1; k < 10; ++k)
        if ((int)blockIdx.x >= q.first[k]) {
            c = 9 - k;
            f0 = q.first[k];
            f1 = q.first[k + 1];
            o0 = q.off[9 - k];
            o1 = q.off[10 - k];
        }
    const int block = (int)blockIdx.x - f0, nblocks = f1 - f0;
    const int32_t count = o1 - o0;
    rows += o0;
    if constexpr (kMode == kModeTry) {
        if (!needs_tables(q.before[c - 6], count))
            cdlp_try_rows(rows, count, col, lab, out, chg, block, nblocks, q.todo + (o0 - q.off[6]), q.now + (c - 6));
        return;
    }
    switch (c) {
        case 0: cdlp_copy_rows(rows, count, lab, out, block, nblocks); break;
        case 1: cdlp_small_rows<2, M>(rows, count, col, lab, out, chg, block, nblocks); break;
        case 2: cdlp_small_rows<4, M>(rows, count, col, lab, out, chg, block, nblocks); break;
        case 3: cdlp_small_rows<8, M>(rows, count, col, lab, out, chg, block, nblocks); break;
        case 4: cdlp_small_rows<16, M>(rows, count, col, lab, out, chg, block, nblocks); break;
        case 5: cdlp_small_rows<32, M>(rows, count, col, lab, out, chg, block, nblocks); break;
        default:
            if constexpr (kMode == kModeMin || kMode == kModeTables) {
                __shared__ int32_t keys[kCdlpThreads / 32][kWarpSlots];
                __shared__ int32_t cnts[kCdlpThreads / 32][kWarpSlots];
                cdlp_warp_rows<M>(rows, count, col, lab, out, chg, block, nblocks, keys[threadIdx.x >> 5],
                                  cnts[threadIdx.x >> 5]);
            }
    }
}

// The rows of a class for a kernel with tables: all of them, or those that
// the try pass listed.
struct CdlpTodo {
    const int4* todo;
    const int32_t* before;  // nullptr: no try pass
    int32_t* now;
    __device__ __forceinline__ bool all(int32_t count) const { return !before || needs_tables(*before, count); }
};

__global__ void __launch_bounds__(kCdlpThreads) cdlp_warp_kernel(const int4* __restrict__ rows, int32_t count,
                                                                 const int32_t* __restrict__ col,
                                                                 const int32_t* __restrict__ lab,
                                                                 int32_t* __restrict__ out, CdlpTodo todo,
                                                                 CdlpChanged chg) {
    __shared__ int32_t keys[kCdlpThreads / 32][kWarpSlots];
    __shared__ int32_t cnts[kCdlpThreads / 32][kWarpSlots];
    const bool all = todo.all(count);
    const int32_t tables =
        cdlp_warp_rows<false>(all ? rows : todo.todo, all ? count : *todo.now, col, lab, out, chg, blockIdx.x,
                              gridDim.x, keys[threadIdx.x >> 5], cnts[threadIdx.x >> 5]);
    if (all && lane_id() == 0 && tables) atomicAdd(todo.now, tables);
}

__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long x, unsigned long long* red) {
    x = warp_max(x);
    if (lane_id() == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long y = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0ull;
        y = warp_max(y);
        if (threadIdx.x == 0) red[0] = y;
    }
    __syncthreads();
    const unsigned long long r = red[0];
    __syncthreads();
    return r;
}

// One block of T threads per row of up to R x T entries (classes 7 to 9), its
// labels in registers; the table (the power of two >= 2 x the row, at least
// 512 slots) lives in 2 x slots ints of dynamic shared memory and is touched
// only by the rows that no label leads.  kMin: the row's smallest label.
template <bool kMin, int R, int T>
__global__ void __launch_bounds__(T) cdlp_block_kernel(
    const int4* __restrict__ rows, int32_t count, const int32_t* __restrict__ col,
    const int32_t* __restrict__ lab, int32_t* __restrict__ out, uint32_t slots, CdlpTodo todo,
    CdlpChanged chg) {
    extern __shared__ int32_t smem[];
    __shared__ unsigned long long red[32];
    __shared__ int32_t s_lead, s_held[2];
    int32_t* K = smem;
    int32_t* C = smem + slots;
    const bool check = !kMin && chg.on();
    const bool all = kMin || todo.all(count);
    if (!all) {
        rows = todo.todo;
        count = *todo.now;
    }
    int32_t tables = 0;  // rows that needed one
    int par = 0;
    if (threadIdx.x < 2) s_held[threadIdx.x] = 0;
    for (int64_t i = blockIdx.x; i < count; i += gridDim.x) {
        const int4 ri = rows[i];
        const int32_t v = ri.x, b = ri.y, e = ri.z;
        int32_t x[R];
        load_cols(x, col, b, e, T, (int)threadIdx.x);
        if (check && !__syncthreads_or(chg.any(x))) {
            if (threadIdx.x == 0) out[v] = lab[v];
            continue;
        }
        gather_labels(x, lab);
        if (kMin) {
            unsigned m = 0xffffffffu;
#pragma unroll
            for (int r = 0; r < R; ++r) m = min(m, (unsigned)x[r]);
            const unsigned long long best = block_max_u64((unsigned long long)(0xffffffffu - m), red);
            if (threadIdx.x == 0) out[v] = (int32_t)(0xffffffffu - (unsigned)best);
            continue;
        }
        if (threadIdx.x < 32) {  // the row holds over 256 entries: a full warp of labels
            const int32_t l = leading_label(x[0]);
            if (threadIdx.x == 0) s_lead = l;
        }
        __syncthreads();
        const int32_t lead = s_lead;
        const int32_t c = count_label(x, lead);
        if (lane_id() == 0 && c) atomicAdd(&s_held[par], c);
        __syncthreads();
        const int32_t held = s_held[par];
        par ^= 1;
        if (threadIdx.x == 0) s_held[par] = 0;  // the next row's; read last before this row's first barrier
        if (2 * held > e - b) {
            if (threadIdx.x == 0) out[v] = lead;
            continue;
        }
        uint32_t cap = 512;
        while (cap < 2u * (uint32_t)(e - b) && cap < slots) cap <<= 1;
        for (uint32_t s = threadIdx.x; s < cap; s += blockDim.x) {
            K[s] = kEmpty;
            C[s] = 0;
        }
        __syncthreads();
        unsigned long long best = insert_labels(K, C, cap, x, lead);
        // Also orders this row's inserts before the next row's clearing.
        best = block_max_u64(best, red);
        if (threadIdx.x == 0) {
            const unsigned long long key = pack_best((uint32_t)held, lead);
            out[v] = unpack_label(best > key ? best : key);
            ++tables;
        }
    }
    if (!kMin && all && tables && todo.before) atomicAdd(todo.now, tables);
}

// Global tables hold slot h as one word, label << 32 | count, empty =
// kSlotEmpty (label kEmpty, count 0): a probe, its count and the later read
// touch one 8-byte word, and a count is added with one 64-bit atomic that
// cannot carry into the label (counts stay below 2^31).
constexpr unsigned long long kSlotEmpty = 0xFFFFFFFF00000000ull;

// Adds cnt to label x in a table of cap slots (cap > 2 x the labels it can
// hold, so a free slot is always reached), probing from slot h.  Sets key to
// (count after this add, label), as table_add returns it, and
// returns the slot when this call claimed it for x, else -1.
__device__ __forceinline__ int32_t global_add_from(unsigned long long* T, uint32_t cap, uint32_t h, int32_t x,
                                                   int32_t cnt, unsigned long long& key) {
    const unsigned long long mine = ((unsigned long long)(uint32_t)x << 32) | (uint32_t)cnt;
    while (true) {
        const unsigned long long cur = atomicCAS(T + h, kSlotEmpty, mine);
        if (cur == kSlotEmpty) {
            key = pack_best((uint32_t)cnt, x);
            return (int32_t)h;
        }
        if ((uint32_t)(cur >> 32) == (uint32_t)x) {
            const unsigned long long old = atomicAdd(T + h, (unsigned long long)cnt);
            key = pack_best((uint32_t)old + (uint32_t)cnt, x);
            return -1;
        }
        h = (h + 1) & (cap - 1);
    }
}

// Chunked-class row i owns pool[tab_off[i] ...] (tab_off even): cap slot
// words, then the list of claimed slots (up to d).  chunks[2k], chunks[2k+1]
// = row index i and the chunk's first entry within the row (a multiple of
// kChunk).
struct LongRow {
    int32_t v, b, d;
    uint32_t cap;
    unsigned long long* T;
    int32_t* L;
};
__device__ __forceinline__ LongRow long_row(const int4* rows, int32_t* pool,
                                            const int64_t* tab_off, int32_t i) {
    LongRow r;
    const int4 ri = rows[i];
    r.v = ri.x;
    r.b = ri.y;
    r.d = ri.z - ri.y;
    r.cap = global_cap(r.d);
    r.T = reinterpret_cast<unsigned long long*>(pool + tab_off[i]);
    r.L = reinterpret_cast<int32_t*>(r.T + r.cap);
    return r;
}

// Called by thread 0 of a block that has finished its chunk of row i with the
// chunk's best (count, -label) key: folds it into best[i]; the row's last
// chunk writes the label, keeps its count in lead[i].x and resets done[i] and
// best[i].
__device__ __forceinline__ void chunk_done(const LongRow& r, int32_t i, unsigned long long b, int32_t* done,
                                           unsigned long long* best, int2* lead, int32_t* out) {
    if (b) atomicMax(best + i, b);
    __threadfence();
    const int32_t nchunks = (r.d + kChunk - 1) / kChunk;
    if (atomicAdd(done + i, 1) == nchunks - 1) {
        __threadfence();
        const unsigned long long won = atomicExch(best + i, 0ull);
        out[r.v] = unpack_label(won);
        lead[i].x = (int32_t)(won >> 32);
        done[i] = 0;
    }
}

// Before the count pass: rows whose last winner held over a quarter of them
// are tried for a label that holds more than half (the leading one of the
// row's first 32 entries), which needs no table.  lead[i] = {the last
// winner's count, the iteration (from 1) whose label this pass wrote}; held[i]
// sums the chunks' matches (zero between iterations).  seen[k] = {label, how
// often chunk k holds it, the iteration that found so}: a chunk counted in the
// last iteration and without a changed vertex since holds as many now.
__global__ void __launch_bounds__(kCdlpThreads) cdlp_chunk_lead_kernel(
    const int4* __restrict__ rows, const int32_t* __restrict__ col, const int32_t* __restrict__ lab,
    const int32_t* __restrict__ chunks, int32_t nch, int32_t* done, int32_t* held, int2* lead,
    int4* seen, int32_t iter, int32_t* __restrict__ out, CdlpChanged chg) {
    const bool check = chg.on();
    __shared__ int32_t s_lead, s_held;
    for (int64_t k = blockIdx.x; k < nch; k += gridDim.x) {
        const int32_t i = chunks[2 * k];
        const int4 ri = rows[i];
        const int32_t d = ri.z - ri.y;
        if (4 * (int64_t)__ldcg(&lead[i].x) <= d) continue;
        const int32_t b = ri.y + chunks[2 * k + 1];
        const int32_t e = (int32_t)min((int64_t)b + kChunk, (int64_t)ri.z);
        int32_t x[kChunk / kCdlpThreads];
        load_cols(x, col, b, e, kCdlpThreads, (int)threadIdx.x);
        const int4 was = seen[k];
        if (threadIdx.x < 32) {
            const int32_t l = leading_label(lab[col[ri.y + threadIdx.x]]);
            if (threadIdx.x == 0) {
                s_lead = l;
                s_held = 0;
            }
        }
        __syncthreads();
        const int32_t want = s_lead;
        if (check && was.z == iter - 1 && was.x == want && !__syncthreads_or(chg.any(x))) {
            if (threadIdx.x == 0) s_held = was.y;
        } else {
            gather_labels(x, lab);
            const int32_t c = count_label(x, want);
            if (lane_id() == 0 && c) atomicAdd(&s_held, c);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            seen[k] = make_int4(want, s_held, iter, 0);
            atomicAdd(held + i, s_held);
            __threadfence();
            if (atomicAdd(done + i, 1) == (d + kChunk - 1) / kChunk - 1) {
                __threadfence();
                const int32_t h = atomicExch(held + i, 0);
                done[i] = 0;
                if (2 * (int64_t)h > d) {
                    out[ri.x] = want;
                    lead[i].y = iter;
                    lead[i].x = h;
                }
            }
        }
        __syncthreads();
    }
}

// One iteration of a chunked-class row, per chunk: count the chunk's labels
// in shared memory, then add each distinct (label, count) to the row's
// global table, keeping the largest key the adds return (the row's answer once
// every chunk has added, as in table_add).  Slots claimed here are
// appended to the row's list (one atomic per warp on occ[i]) for the reset
// pass.
__global__ void __launch_bounds__(kCdlpThreads) cdlp_chunk_count_kernel(
    const int4* __restrict__ rows, const int32_t* __restrict__ col,
    const int32_t* __restrict__ lab, const int32_t* __restrict__ chunks, int32_t nch, int32_t* pool,
    const int64_t* __restrict__ tab_off, int32_t* occ, int32_t* done, unsigned long long* best, int2* lead,
    int32_t iter, int32_t* __restrict__ out) {
    extern __shared__ int32_t smem[];
    __shared__ unsigned long long red[32];
    int32_t* K = smem;
    int32_t* C = smem + kChunkSlots;
    for (int64_t k = blockIdx.x; k < nch; k += gridDim.x) {
        const int32_t i = chunks[2 * k];
        if (lead[i].y == iter) continue;  // its label is written
        const LongRow r = long_row(rows, pool, tab_off, i);
        const int32_t b = r.b + chunks[2 * k + 1];
        const int32_t e = (int32_t)min((int64_t)b + kChunk, (int64_t)r.b + r.d);
        int32_t x[kChunk / kCdlpThreads];
        load_cols(x, col, b, e, kCdlpThreads, (int)threadIdx.x);
        gather_labels(x, lab);
        uint32_t cap = 512;
        while (cap < 2u * (uint32_t)(e - b) && cap < (uint32_t)kChunkSlots) cap <<= 1;
        for (uint32_t s = threadIdx.x; s < cap; s += blockDim.x) {
            K[s] = kEmpty;
            C[s] = 0;
        }
        __syncthreads();
        // Each warp's leading label goes in once for all of its entries.
        const int32_t first = leading_label(x[0]);
        const int32_t held = count_label(x, first);
        insert_labels(K, C, cap, x, first);
        if (lane_id() == 0 && first >= 0) table_add(K, C, cap, first, held);
        __syncthreads();
        // The chunk's distinct labels go to the global table kF per thread at
        // a time: the kF home-slot CASes issue together, then the adds for
        // labels found there, and only a slot held by another label is probed
        // one step at a time.  cap is a multiple of the block size: every
        // warp runs every round.
        constexpr int kF = 4;
        unsigned long long mx = 0;
        for (uint32_t s0 = 0; s0 < cap; s0 += kF * blockDim.x) {
            int32_t x[kF], c[kF];
            uint32_t h[kF];
            unsigned long long cur[kF], old[kF];
#pragma unroll
            for (int q = 0; q < kF; ++q) {
                const uint32_t s = s0 + q * blockDim.x + threadIdx.x;
                x[q] = s < cap ? K[s] : kEmpty;
                c[q] = s < cap ? C[s] : 0;
                h[q] = hash_label(x[q]) & (r.cap - 1);
                cur[q] = x[q] != kEmpty ? atomicCAS(r.T + h[q], kSlotEmpty,
                                                    ((unsigned long long)(uint32_t)x[q] << 32) | (uint32_t)c[q])
                                        : kSlotEmpty;
            }
#pragma unroll
            for (int q = 0; q < kF; ++q) {
                old[q] = 0;
                if (x[q] != kEmpty && cur[q] != kSlotEmpty && (uint32_t)(cur[q] >> 32) == (uint32_t)x[q])
                    old[q] = atomicAdd(r.T + h[q], (unsigned long long)c[q]);
            }
#pragma unroll
            for (int q = 0; q < kF; ++q) {
                if (s0 + q * blockDim.x >= cap) break;
                int32_t claimed = -1;
                unsigned long long key = 0;
                if (x[q] != kEmpty) {
                    if (cur[q] == kSlotEmpty) {
                        claimed = (int32_t)h[q];
                        key = pack_best((uint32_t)c[q], x[q]);
                    } else if ((uint32_t)(cur[q] >> 32) == (uint32_t)x[q]) {
                        key = pack_best((uint32_t)old[q] + (uint32_t)c[q], x[q]);
                    } else {
                        claimed = global_add_from(r.T, r.cap, (h[q] + 1) & (r.cap - 1), x[q], c[q], key);
                    }
                }
                mx = key > mx ? key : mx;
                const unsigned m = __ballot_sync(0xffffffffu, claimed >= 0);
                if (m) {
                    int32_t base = 0;
                    if (lane_id() == 0) base = atomicAdd(occ + i, __popc(m));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (claimed >= 0) r.L[base + __popc(m & ((1u << lane_id()) - 1u))] = claimed;
                }
            }
        }
        // Also orders this chunk's table reads before the next chunk's clearing.
        mx = block_max_u64(mx, red);
        if (threadIdx.x == 0) chunk_done(r, i, mx, done, best, lead, out);
    }
}

// After the count pass: empties the slots the pass claimed, by writes only.
// A sparse table (at most cap / 8 claims, the usual case once labels
// converge) is reset through its claim list, chunk k taking list entries
// [j0, j0 + kChunk); a dense one in slot order, chunk k taking the k-th share
// of the slots.  The row's last chunk resets occ[i] and done[i].
__global__ void __launch_bounds__(kCdlpThreads) cdlp_chunk_reset_kernel(
    const int4* __restrict__ rows, const int32_t* __restrict__ chunks,
    int32_t nch, int32_t* pool, const int64_t* __restrict__ tab_off, int32_t* occ, int32_t* done,
    const int2* __restrict__ lead, int32_t iter) {
    for (int64_t k = blockIdx.x; k < nch; k += gridDim.x) {
        const int32_t i = chunks[2 * k];
        if (lead[i].y == iter) continue;  // nothing was counted
        const LongRow r = long_row(rows, pool, tab_off, i);
        const int32_t j0 = chunks[2 * k + 1];
        const int32_t claims = __ldcg(occ + i);
        const uint32_t nchunks = (uint32_t)(r.d + kChunk - 1) / kChunk;
        if ((uint32_t)claims > r.cap / 8) {
            const uint32_t per = (r.cap + nchunks - 1) / nchunks;
            const uint32_t s0 = (uint32_t)(j0 / kChunk) * per;
            const uint32_t s1 = min(s0 + per, r.cap);
            for (uint32_t s = s0 + threadIdx.x; s < s1; s += blockDim.x) r.T[s] = kSlotEmpty;
        } else {
            const int32_t j1 = (int32_t)min((int64_t)j0 + kChunk, (int64_t)claims);
            for (int32_t j = j0 + threadIdx.x; j < j1; j += blockDim.x) r.T[__ldcg(r.L + j)] = kSlotEmpty;
        }
        __syncthreads();  // every thread has read occ[i] before it can be reset
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(done + i, 1) == (int32_t)nchunks - 1) {
                occ[i] = 0;
                done[i] = 0;
            }
        }
    }
}

// First iteration (labels distinct, no repeated entries): each chunk's
// smallest label, folded over the row's chunks as in the pick pass.
__global__ void __launch_bounds__(kCdlpThreads) cdlp_chunk_min_kernel(
    const int4* __restrict__ rows, const int32_t* __restrict__ col,
    const int32_t* __restrict__ lab, const int32_t* __restrict__ chunks, int32_t nch, int32_t* pool,
    const int64_t* __restrict__ tab_off, int32_t* done, unsigned long long* best, int2* lead,
    int32_t* __restrict__ out) {
    __shared__ unsigned long long red[32];
    for (int64_t k = blockIdx.x; k < nch; k += gridDim.x) {
        const int32_t i = chunks[2 * k];
        const LongRow r = long_row(rows, pool, tab_off, i);
        const int32_t b = r.b + chunks[2 * k + 1];
        const int32_t e = (int32_t)min((int64_t)b + kChunk, (int64_t)r.b + r.d);
        unsigned long long m = 0;
        for (int32_t j = b + threadIdx.x; j < e; j += blockDim.x) {
            const unsigned long long key = pack_best(1, lab[col[j]]);
            m = key > m ? key : m;
        }
        m = block_max_u64(m, red);
        if (threadIdx.x == 0) chunk_done(r, i, m, done, best, lead, out);
    }
}

// Chunked-class rows: degrees for the host's table layout.
__global__ void cdlp_long_degrees_kernel(const int4* __restrict__ rows, int32_t count, int32_t* deg) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        deg[i] = rows[i].z - rows[i].y;
    }
}

// Block per chunked-class row: every slot empty.
__global__ void cdlp_pool_clear_kernel(const int4* __restrict__ rows, int32_t count, int32_t* pool,
                                       const int64_t* __restrict__ tab_off) {
    for (int64_t i = blockIdx.x; i < count; i += gridDim.x) {
        const LongRow r = long_row(rows, pool, tab_off, (int32_t)i);
        for (uint32_t s = threadIdx.x; s < r.cap; s += blockDim.x) r.T[s] = kSlotEmpty;
    }
}

}  // namespace

// init_labels (device, may be NULL = vertex ids): starting label values.
// first_min: the rows repeat no entry and the starting labels are distinct,
// so the first iteration is a minimum over each row's labels.
int cdlp_run(ghb_workspace* ws, int32_t n, const int32_t* rp, const int32_t* col, int32_t iterations,
             int32_t* labels, const int32_t* init_labels, bool first_min) {
    cudaStream_t st = ws->stream;
    int32_t* hp = reinterpret_cast<int32_t*>(ws->host_pinned);

    // Pass 1: class sizes.
    Carver pre(nullptr);
    pre.take<int32_t>(16);
    GHB_TRY(ws_reserve(ws, pre.off + (size_t)n * 4 * 3 + 4096));
    int32_t* counts = reinterpret_cast<int32_t*>(ws->scratch);
    GHB_CUDA_TRY(cudaMemsetAsync(counts, 0, 16 * sizeof(int32_t), st));
    GHB_TRY(launch(ws, cdlp_count_classes_kernel, dim3(grid_for(n, kCdlpThreads, ws->num_sms * 8)),
                   dim3(kCdlpThreads), 0, n, rp, counts));
    GHB_CUDA_TRY(cudaMemcpyAsync(hp, counts, 16 * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    GHB_CUDA_TRY(cudaStreamSynchronize(st));
    int32_t cls[kCdlpClasses], off[kCdlpClasses + 1];
    off[0] = 0;
    for (int k = 0; k < kCdlpClasses; ++k) {
        cls[k] = hp[k];
        off[k + 1] = off[k] + cls[k];
    }
    // Chunked-class tables: (label, count) pairs for the power of two >= 2 d
    // slots, then the claimed-slot list of d ints (rounded up to even), so
    // fewer than 9 ints per entry plus one per row.
    const int32_t nlong = cls[10];
    const int64_t long_entries = hp[kSumLongSlot], entries = hp[kSumSlot];
    const int64_t pool_bound = nlong > 0 ? 9 * long_entries + nlong + 16 : 1;
    const int64_t chunk_bound = long_entries / kChunk + nlong + 1;
    Carver sizing(nullptr);
    sizing.take<int32_t>(16);
    sizing.take<int32_t>(16);
    sizing.take<int4>(n);
    sizing.take<int32_t>(n);
    sizing.take<int32_t>(pool_bound);
    sizing.take<int64_t>((size_t)nlong + 1);
    sizing.take<int32_t>(2 * chunk_bound);
    sizing.take<int32_t>((size_t)nlong + 1);
    sizing.take<int32_t>((size_t)nlong + 1);
    sizing.take<unsigned long long>((size_t)nlong + 1);
    sizing.take<int32_t>((size_t)nlong + 1);
    sizing.take<int2>((size_t)nlong + 1);
    sizing.take<int4>(chunk_bound);
    sizing.take<uint32_t>((size_t)n / 32 + 1);
    sizing.take<int32_t>(iterations + 1);
    sizing.take<int32_t>(4 * ((size_t)iterations + 1));
    sizing.take<int4>((size_t)(off[10] - off[6]) + 1);
    GHB_TRY(ws_reserve(ws, sizing.off));
    Carver c(ws->scratch);
    counts = c.take<int32_t>(16);
    int32_t* cursor = c.take<int32_t>(16);
    int4* rows = c.take<int4>(n);
    int32_t* other = c.take<int32_t>(n);
    int32_t* pool = c.take<int32_t>(pool_bound);
    int64_t* tab_off = c.take<int64_t>((size_t)nlong + 1);
    int32_t* chunks = c.take<int32_t>(2 * chunk_bound);
    int32_t* occ = c.take<int32_t>((size_t)nlong + 1);
    int32_t* done = c.take<int32_t>((size_t)nlong + 1);
    unsigned long long* best = c.take<unsigned long long>((size_t)nlong + 1);
    int32_t* held = c.take<int32_t>((size_t)nlong + 1);
    int2* lead = c.take<int2>((size_t)nlong + 1);
    int4* seen = c.take<int4>(chunk_bound);
    uint32_t* changed = c.take<uint32_t>((size_t)n / 32 + 1);
    int32_t* nchanged = c.take<int32_t>(iterations + 1);
    int32_t* ntodo = c.take<int32_t>(4 * ((size_t)iterations + 1));
    int4* todo = c.take<int4>((size_t)(off[10] - off[6]) + 1);

    for (int k = 0; k < kCdlpClasses; ++k) hp[k] = off[k];
    GHB_CUDA_TRY(cudaMemcpyAsync(cursor, hp, kCdlpClasses * sizeof(int32_t), cudaMemcpyHostToDevice, st));
    GHB_TRY(launch(ws, cdlp_fill_classes_kernel, dim3(grid_for(n, kFillRows * kCdlpThreads, ws->num_sms * 8)),
                   dim3(kCdlpThreads), 0, n, rp, cursor, rows));
    const int4* long_rows = rows + off[10];
    int32_t nch = 0;
    if (nlong > 0) {
        // Table offsets and the chunk list on the host (a few thousand rows),
        // then empty tables and zero counters.
        GHB_TRY(launch(ws, cdlp_long_degrees_kernel, dim3(grid_for(nlong, 256, ws->num_sms)), dim3(256), 0,
                       long_rows, nlong, occ));
        std::vector<int32_t> deg((size_t)nlong);
        GHB_CUDA_TRY(cudaMemcpyAsync(deg.data(), occ, sizeof(int32_t) * nlong, cudaMemcpyDeviceToHost, st));
        GHB_CUDA_TRY(cudaStreamSynchronize(st));
        std::vector<int64_t> toff((size_t)nlong + 1);
        std::vector<int32_t> ch;
        ch.reserve(2 * (size_t)chunk_bound);
        int64_t acc = 0;
        for (int32_t i = 0; i < nlong; ++i) {
            // global_cap needs 2 d <= 2^31.
            GHB_REQUIRE(deg[i] <= (1 << 30), "CDLP: a row holds more than 2^30 entries");
            toff[i] = acc;
            acc += 2 * (int64_t)global_cap(deg[i]) + ((deg[i] + 1) & ~1);  // keeps every tab_off even
            for (int64_t j = 0; j < deg[i]; j += kChunk) {
                ch.push_back(i);
                ch.push_back((int32_t)j);
            }
        }
        toff[nlong] = acc;
        nch = (int32_t)(ch.size() / 2);
        GHB_REQUIRE(acc <= pool_bound && nch <= chunk_bound, "CDLP table pool bound");
        GHB_CUDA_TRY(cudaMemcpyAsync(tab_off, toff.data(), sizeof(int64_t) * (nlong + 1), cudaMemcpyHostToDevice, st));
        GHB_CUDA_TRY(cudaMemcpyAsync(chunks, ch.data(), sizeof(int32_t) * ch.size(), cudaMemcpyHostToDevice, st));
        // occ, done, best, held, lead and seen lie behind one another.
        GHB_CUDA_TRY(cudaMemsetAsync(occ, 0, (size_t)(reinterpret_cast<char*>(seen + nch) - reinterpret_cast<char*>(occ)), st));
        GHB_TRY(launch(ws, cdlp_pool_clear_kernel, dim3(grid_for(nlong, 1, ws->num_sms * 8)), dim3(256), 0, long_rows,
                       nlong, pool, (const int64_t*)tab_off));
        GHB_CUDA_TRY(cudaStreamSynchronize(st));  // toff and ch are read by the copies above
    }
    if (init_labels)
        GHB_CUDA_TRY(cudaMemcpyAsync(labels, init_labels, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st));
    else
        GHB_TRY(launch(ws, cdlp_iota_kernel, dim3(grid_for(n, 256, ws->num_sms * 8)), dim3(256), 0, labels, n));

    // Shared-memory classes: as many blocks as fit each SM.
    const size_t small_smem = 2 * kSmallBlockSlots * sizeof(int32_t), big_smem = 2 * kBlockSlots * sizeof(int32_t);
    const size_t chunk_smem = 2 * kChunkSlots * sizeof(int32_t), mid_smem = 2 * kMidBlockSlots * sizeof(int32_t);
    GHB_CUDA_TRY(cudaFuncSetAttribute(cdlp_block_kernel<false, 8, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)big_smem));
    GHB_CUDA_TRY(cudaFuncSetAttribute(cdlp_chunk_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)chunk_smem));
    int per_sm_small = 0, per_sm_mid = 0, per_sm_big = 0, per_sm_chunk = 0;
    GHB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_small, cdlp_block_kernel<false, 4, 256>, kCdlpThreads,
                                                               small_smem));
    GHB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_mid, cdlp_block_kernel<false, 8, 256>, kCdlpThreads,
                                                               mid_smem));
    GHB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_big, cdlp_block_kernel<false, 8, 512>, 512,
                                                               big_smem));
    GHB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_chunk, cdlp_chunk_count_kernel, kCdlpThreads,
                                                               chunk_smem));
    const unsigned g_small = ws->num_sms * std::max(1, per_sm_small);
    const unsigned g_mid = ws->num_sms * std::max(1, per_sm_mid);
    const unsigned g_big = ws->num_sms * std::max(1, per_sm_big);
    const unsigned g_chunk = ws->num_sms * std::max(1, per_sm_chunk);
    const unsigned g = ws->num_sms * 8;

    // Large inputs: unchanged neighbourhoods and led rows apart from the rows
    // that need tables.  The extra launches of an iteration cost a small input
    // more than they save.
    const bool large = n >= kCheckRows && iterations > 2;
    // The bits cost a pass over both label arrays an iteration and a look an entry,
    // and save label gathers once few labels move: nothing below 6 entries a
    // vertex (with and without, 30 iterations: 700 x 700 grid 588 and 455 us, uniform
    // of 2^20 vertices and 4 entries 1,176 and 1,032, communities of 5.6 1,315 and
    // 1,268; uniform of 8 1,627 and 1,945, of 12 2,391 and 3,250).
    const bool bits = large && entries >= 6ll * n;
    if (large) {
        // nchanged and ntodo lie behind one another.  Before the first iteration
        // that counts: as if every row had needed its table.
        GHB_CUDA_TRY(cudaMemsetAsync(nchanged, 0, (size_t)(reinterpret_cast<char*>(ntodo + 4 * ((size_t)iterations + 1)) -
                                                           reinterpret_cast<char*>(nchanged)), st));
        GHB_CUDA_TRY(cudaMemsetAsync(ntodo + (first_min ? 4 : 0), 0x7f, sizeof(int32_t) * 4, st));
    }
    auto light_plan = [&](int from, int classes) {
        CdlpLight q = {};
        for (int k = 0; k < 10; ++k) {
            const int c = 9 - k;
            const int64_t threads = (int64_t)cls[c] * (c == 0 ? 1 : c < 6 ? 1 << c : 32);
            q.off[c] = off[c];
            q.first[k + 1] =
                q.first[k] + (c >= from && c < classes && cls[c] ? (int32_t)grid_for(threads, kCdlpThreads, g) : 0);
        }
        q.off[10] = off[10];
        return q;
    };
    // Rows without entries keep their labels: once both buffers hold them
    // (after two iterations) class 0 is left out.
    const int classes = large ? 6 : 7;
    const CdlpLight first = light_plan(0, 7), light = light_plan(0, classes), later = light_plan(1, classes);
    CdlpLight longer = light_plan(6, 10);

    // Iteration it reads cur and writes nxt.  kMin (first iteration over
    // distinct labels): each row's smallest label.
    auto iteration = [&](auto min_tag, int it, const int32_t* cur, int32_t* nxt, CdlpChanged chg) -> int {
        constexpr bool M = decltype(min_tag)::value;
        const int4* R = rows;
        const dim3 block(kCdlpThreads);
        const bool tries = large && !M;
        const CdlpLight q = M ? first : it >= 2 ? later : light;
        // Class 6 + k: listed rows, their number last time and this time.
        auto list = [&](int k) {
            return tries ? CdlpTodo{todo + (off[6 + k] - off[6]), ntodo + 4 * it + k, ntodo + 4 * (it + 1) + k}
                         : CdlpTodo{nullptr, nullptr, nullptr};
        };
        const dim3 grid(q.first[10]);
        if (grid.x)
            GHB_TRY(launch(ws, M ? cdlp_light_kernel<kModeMin> : tries ? cdlp_light_kernel<kModeSmall> : cdlp_light_kernel<kModeTables>,
                           grid, block, 0, R, q, col, cur, nxt, chg));
        if (tries && longer.first[10]) {
            longer.todo = todo;
            longer.before = ntodo + 4 * it;
            longer.now = ntodo + 4 * (it + 1);
            GHB_TRY(launch(ws, cdlp_light_kernel<kModeTry>, dim3(longer.first[10]), block, 0, R, longer, col, cur, nxt, chg));
        }
        if (tries && cls[6])
            GHB_TRY(launch(ws, cdlp_warp_kernel, dim3(grid_for((int64_t)cls[6] * 32, kCdlpThreads, ws->num_sms * 7)), block, 0,
                           R + off[6], cls[6], col, cur, nxt, list(0), chg));
        if (M) {
            if (cls[7]) GHB_TRY(launch(ws, cdlp_block_kernel<true, 4, 256>, dim3(grid_for(cls[7], 1, g)), block, 0, R + off[7], cls[7], col, cur, nxt, 0u, list(0), chg));
            if (cls[8]) GHB_TRY(launch(ws, cdlp_block_kernel<true, 8, 256>, dim3(grid_for(cls[8], 1, g)), block, 0, R + off[8], cls[8], col, cur, nxt, 0u, list(0), chg));
            if (cls[9]) GHB_TRY(launch(ws, cdlp_block_kernel<true, 8, 512>, dim3(grid_for(cls[9], 1, g)), dim3(512), 0, R + off[9], cls[9], col, cur, nxt, 0u, list(0), chg));
            if (nlong) GHB_TRY(launch(ws, cdlp_chunk_min_kernel, dim3(grid_for(nch, 1, g)), block, 0, long_rows, col, cur, (const int32_t*)chunks, nch, pool, (const int64_t*)tab_off, done, best, lead, nxt));
            return GHB_OK;
        }
        if (cls[7]) GHB_TRY(launch(ws, cdlp_block_kernel<false, 4, 256>, dim3(grid_for(cls[7], 1, g_small)), block, small_smem, R + off[7], cls[7], col, cur, nxt, (uint32_t)kSmallBlockSlots, list(1), chg));
        if (cls[8]) GHB_TRY(launch(ws, cdlp_block_kernel<false, 8, 256>, dim3(grid_for(cls[8], 1, g_mid)), block, mid_smem, R + off[8], cls[8], col, cur, nxt, (uint32_t)kMidBlockSlots, list(2), chg));
        if (cls[9]) GHB_TRY(launch(ws, cdlp_block_kernel<false, 8, 512>, dim3(grid_for(cls[9], 1, g_big)), dim3(512), big_smem, R + off[9], cls[9], col, cur, nxt, (uint32_t)kBlockSlots, list(3), chg));
        if (nlong) {
            GHB_TRY(launch(ws, cdlp_chunk_lead_kernel, dim3(grid_for(nch, 1, g)), block, 0, long_rows, col, cur, (const int32_t*)chunks, nch, done, held, lead, seen, it + 1, nxt, chg));
            GHB_TRY(launch(ws, cdlp_chunk_count_kernel, dim3(grid_for(nch, 1, g_chunk)), block, chunk_smem, long_rows, col, cur, (const int32_t*)chunks, nch, pool, (const int64_t*)tab_off, occ, done, best, lead, it + 1, nxt));
            GHB_TRY(launch(ws, cdlp_chunk_reset_kernel, dim3(grid_for(nch, 1, g)), block, 0, long_rows, (const int32_t*)chunks, nch, pool, (const int64_t*)tab_off, occ, done, (const int2*)lead, it + 1));
        }
        return GHB_OK;
    };

    int32_t* cur = labels;
    int32_t* nxt = other;
    for (int it = 0; it < iterations; ++it) {
        // The bits pay while few labels moved: never behind the first iteration.
        const CdlpChanged chg{bits && it > 1 ? changed : nullptr, nchanged + (it > 0 ? it - 1 : 0), n / 16};
        if (it == 0 && first_min)
            GHB_TRY(iteration(std::true_type{}, it, cur, nxt, chg));
        else
            GHB_TRY(iteration(std::false_type{}, it, cur, nxt, chg));
        if (bits && it > 0 && it + 1 < iterations)
            GHB_TRY(launch(ws, cdlp_changed_kernel, dim3(grid_for(n, kCdlpThreads, g)), dim3(kCdlpThreads), 0, n,
                           (const int32_t*)cur, (const int32_t*)nxt, changed, nchanged + it));
        std::swap(cur, nxt);
    }
    if (cur != labels)
        GHB_CUDA_TRY(cudaMemcpyAsync(labels, cur, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st));
    return GHB_OK;
}

}  // namespace ghb

using namespace ghb;

extern "C" int ghb_cdlp(ghb_workspace* ws, int32_t n, const int32_t* all_rowptr, const int32_t* all_col,
                        int32_t iterations, int32_t* labels) {
    ws = ws_resolve(ws);
    GHB_REQUIRE(ws, "no workspace");
    GHB_REQUIRE(n >= 1, "n must be >= 1");
    GHB_REQUIRE(all_rowptr && labels, "NULL argument");
    GHB_REQUIRE(iterations >= 0, "iterations < 0");
    return cdlp_run(ws, n, all_rowptr, all_col, iterations, labels, nullptr, false);
}
