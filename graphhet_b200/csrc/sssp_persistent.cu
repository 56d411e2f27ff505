// Whole single-source shortest-path traversal in one cooperative launch.
//
// The host-driven delta-stepping (sssp.cu) pays a host round trip and
// several launches per relaxation round, like the reference's
// frontier loop (GPU_SSSP_csr.cuh:286-307, a device-to-host copy of the
// queue length per iteration).  Here every round runs inside one launch and
// the grid meets at a bounded barrier between passes; every block then
// derives the next pass from the same counters.  Passes over small queues run
// on block 0 alone, the others waiting at one barrier:
//
//   LIGHT  relax the light range (entries with w < delta of the weight-sorted
//          rows; the whole row when there is no split) of every near-queue
//          vertex.  An improvement below the bucket's end queues the vertex
//          for the next LIGHT pass, one at or above it goes to the far list.
//          Each queued vertex also joins R, the bucket's settled set.
//   HEAVY  relax the heavy range (w >= delta) of every vertex of R once.
//   CHUNK  after a LIGHT or HEAVY pass that met rows of more than kSpDirect
//          entries: those rows, cut into kSpChunk-entry chunks, a chunk per
//          warp, in the same round (same stamps, same next queue).
//   SPLIT  move the far list's entries below the next bucket's end into the
//          near queue; drop entries already settled; keep the rest.
//
// Grid passes stage what they append in shared memory (SpStage).
//
// The next bucket's end follows the smallest pending far distance
// (kept in shared memory per block, one global atomic per block and pass),
// so empty buckets cost nothing.
//
// Results are the least fixpoint of d[v] = min_u fl(d[u] + w): any
// relaxation order reaches it bit for bit (see sssp.cu), so they equal the
// CPU Dijkstra's (CPU_shortest_paths.hpp:19-64).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "graph.cuh"
#include "row_math.cuh"

namespace ghb {

// Rows of up to kSpDirect entries are relaxed where the queue hands them to a
// warp; longer ones are cut into kSpChunk-entry chunks that a CHUNK pass, in
// the same round, spreads over every warp (a warp walking a few 1,024-entry
// rows while the rest of the grid waits at the barrier was the bottleneck).
// Chunks are one step of a warp, kSpBatch x 32 entries: RMAT-16 0.58 ms with
// 256 and 0.54 with 128, RMAT-18 on the caller's ids 0.84 and 0.80, uniform
// graphs alike; 512 costs RMAT-20 raw 1.42 -> 1.70.
constexpr int32_t kSpDirect = 64;
constexpr int32_t kSpChunk = 128;
constexpr int kSsspThreads = 512;
// Passes over small queues run on block 0 alone (see sssp_persistent_kernel):
// its queues' first kSoloQueue entries lie in shared memory, and it hands back
// to the grid after kSoloTurns passes at the latest.
constexpr int32_t kSoloQueue = 2048;
constexpr int32_t kSoloChunks = 32;
// A queue is small up to kSoloEntries entries of mean degree.  1501 x 1999
// grid, the caller's rows from a corner, before the staging below (33 ms with
// it): 30.8 ms with 3072, 35.8 with 6144 and 40.3 with 12288 (one block then takes
// several turns of 512 rows per pass), 59.7 with every pass on the grid and its
// decision read back through L2 (300 x 300: 3.3 ms against 9.0).
constexpr int64_t kSoloEntries = 3072;
constexpr int kSoloTurns = 1 << 14;
constexpr unsigned long long kSsspTimeBudgetNs = 120ull * 1000000000ull;  // two minutes

enum SsspMode : int32_t { kLight = 0, kHeavy = 1, kSplit = 2, kDone = 3, kChunk = 4 };

// What a pass appends to.  Three slots by pass number: pass p fills slot
// p % 3, every block reads it after the pass's barrier, and block 0 clears
// slot (p + 1) % 3 during pass p (all blocks read it last before the barrier
// of pass p - 1).
struct SpSlot {
    // A cache line for each: atomics on one line follow each other at about
    // 2 ns, whichever of its words they take.
    alignas(128) int32_t q_tail;   // the next near queue
    alignas(128) int32_t c_tail;   // chunks
    alignas(128) int32_t r_add;    // additions to R
    alignas(128) int32_t far_add;  // additions to the far list
    alignas(128) unsigned long long fmin;  // smallest far distance added (bits)
    alignas(128) unsigned long long examined;
    int32_t stop;                  // the time budget ran out
};

// Where the traversal stands: every block holds it in shared memory and
// derives the next pass from it and the slot just filled, so no block waits
// for another's decision to be written and read back.
struct SpState {
    int32_t mode;         // SsspMode of the current pass
    int32_t solo;         // 1: block 0 runs it alone
    int32_t round;        // stamp of the near queue being filled
    int32_t phase;        // stamp of the far list being filled
    int32_t epoch;        // stamp of R (bumped after every HEAVY pass)
    int32_t nq;           // items of the current queue (near queue, R in HEAVY, far list in SPLIT)
    int32_t nc;           // chunk items of the current (CHUNK) pass
    int32_t qsel;         // near queue buffer read by the current pass
    int32_t chunk_of;     // the pass (LIGHT or HEAVY) whose rows a CHUNK pass finishes
    int32_t fsel;         // far buffer filled (a SPLIT reads the other)
    int32_t q_next;       // near-queue entries filled by a pass whose chunks are still to come
    int32_t r_count, far_count;  // R's and the far list's entries
    int32_t failed;       // a budget ran out
    double thr;           // end of the current bucket
    double new_thr;       // end of the next bucket (SPLIT)
    // Bucket width: the light/heavy split stays at delta; the width of the
    // buckets may move within [width_min, width_max] from one bucket to the
    // next (equal to delta when the width does not adapt).
    double width, width_min, width_max;
    unsigned long long fmin;  // smallest pending far distance (bits; an upper bound on stale entries)
    unsigned long long examined;
    long long passes, light_passes, heavy_passes, splits, chunk_passes;
    long long pass_budget;
    long long lp_mark;              // LIGHT passes before the current bucket
    unsigned long long ex_mark;     // entries examined before the current bucket
    unsigned long long adapt_work;  // a bucket examining fewer entries is small
    int32_t solo_max;               // queues up to this many vertices run on block 0 alone
    int32_t pad;
};

struct SsspRunState {
    unsigned bar_count;  // barrier arrivals (own cache line)
    unsigned pad_a[31];
    unsigned bar_release;  // barrier epochs (own cache line)
    unsigned pad_b[31];
    int32_t status;
    unsigned bar_extra;
    unsigned long long bar_limit_ns;
    unsigned pad_c[28];
    SpSlot slot[3];
    SpState s;  // set by the host; block 0's after a solo run and at the end
};

namespace {

__device__ __forceinline__ double sp_dist(const unsigned long long* d, int32_t v) {
    return __longlong_as_double((long long)__ldcg(d + v));
}

// A queue whose first `cap` entries may lie in shared memory (solo runs).
struct SpQueue {
    int32_t* fast;
    int32_t* mem;
    int32_t cap;
    __device__ __forceinline__ int32_t get(int32_t i) const { return i < cap ? fast[i] : __ldcg(mem + i); }
    __device__ __forceinline__ void put(int32_t i, int32_t v) const {
        if (i < cap) fast[i] = v;
        else mem[i] = v;
    }
};

// What a warp has yet to append in a grid pass, by kind: it writes kSpStage at
// a time behind one atomic on the list's counter, and the block's warps the
// rest behind one at the end of the pass.  With an atomic per step of 128
// entries relaxed and one per long row, the counters' cache line set the
// pace, at 2 ns an atomic: a light pass over 690,000 rows of RMAT-22 took
// 450 us and takes 130, its long rows' 23 M entries 517 and 210, a heavy
// pass of 80 M entries 1,000 and 530.  One source on RMAT-22, resident, 6.1 ->
// 3.0 ms, on the caller's ids 13.2 -> 4.5; RMAT-20 of degree 8 2.7 -> 1.9 and
// 2.8 -> 1.3; uniform, 2^20 vertices of degree 16, 1.11 -> 0.77.  Grids, whose
// passes are mostly solo, give 4 % for the longer code.
enum SpKind : int { kNear = 0, kFar = 1, kSettled = 2, kSpKinds = 3 };
constexpr int kSpStage = 128;
constexpr int kSpWarps = kSsspThreads / 32;
struct SpStage {
    int32_t* buf;  // the warp's kSpKinds x kSpStage words; nullptr: append at once (solo passes)
    int32_t n[kSpKinds];
};

struct SpCtx {
    const int32_t* __restrict__ rp;
    const int32_t* __restrict__ le;  // light ends (nullptr: no light/heavy split)
    const int32_t* __restrict__ col;
    const double* __restrict__ wt;
    unsigned long long* dist;
    int32_t* near_stamp;
    int32_t* far_stamp;
    int32_t* r_stamp;
    int32_t* R;
    SpQueue q_next;
    int32_t* far_cur;
    int4* chunks;
    SpSlot* slot;
    double thr;
    int32_t round, phase, epoch;
    int32_t q_base, r_base, far_base;  // entries that were there before the pass
};

// Entries a lane relaxes per step: their column, weight and distance loads
// are all issued before any compare, so a lane keeps kSpBatch gathers in
// flight instead of one dependent chain.
constexpr int kSpBatch = 4;

// What a thread has found in a pass: entries relaxed (a pass relaxes fewer
// than 2^31) and its smallest far distance (bits).
struct SpFound {
    unsigned exam = 0;
    unsigned long long fmin = ~0ull;
};

template <int KIND>
__device__ __forceinline__ int32_t* sp_tail(const SpCtx& c) {
    return KIND == kNear ? &c.slot->q_tail : KIND == kFar ? &c.slot->far_add : &c.slot->r_add;
}
template <int KIND>
__device__ __forceinline__ int32_t sp_base(const SpCtx& c) {
    return KIND == kNear ? c.q_base : KIND == kFar ? c.far_base : c.r_base;
}
template <int KIND>
__device__ __forceinline__ int32_t* sp_list(const SpCtx& c) {
    return KIND == kNear ? c.q_next.mem : KIND == kFar ? c.far_cur : c.R;
}

// The warp's staged vertices of one kind, to their list from position at.
template <int KIND>
__device__ __forceinline__ void sp_write(const SpCtx& c, SpStage& g, int32_t at) {
    for (int32_t i = lane_id(); i < g.n[KIND]; i += 32) sp_list<KIND>(c)[at + i] = g.buf[KIND * kSpStage + i];
}

// Append v[q] of the lanes in m[q]; every lane of the warp calls it.
template <int KIND, int Q>
__device__ __forceinline__ void sp_append(const SpCtx& c, SpStage& g, const unsigned* m, const int32_t* v) {
    int32_t total = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) total += __popc(m[q]);
    if (total == 0) return;
    const int lane = lane_id();
    const unsigned below = (1u << lane) - 1u;
    int32_t at;
    if (g.buf) {
        static_assert(Q * 32 <= kSpStage, "a step's entries fit an empty buffer");
        if (g.n[KIND] + total > kSpStage) {
            int32_t to = 0;
            if (lane == 0) to = sp_base<KIND>(c) + atomicAdd(sp_tail<KIND>(c), g.n[KIND]);
            __syncwarp();
            sp_write<KIND>(c, g, __shfl_sync(0xffffffffu, to, 0));
            __syncwarp();
            g.n[KIND] = 0;
        }
        at = g.n[KIND];
        g.n[KIND] += total;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            if ((m[q] >> lane) & 1u) g.buf[KIND * kSpStage + at + __popc(m[q] & below)] = v[q];
            at += __popc(m[q]);
        }
        return;
    }
    at = 0;
    if (lane == 0) at = sp_base<KIND>(c) + atomicAdd(sp_tail<KIND>(c), total);
    at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        if ((m[q] >> lane) & 1u) {
            const int32_t i = at + __popc(m[q] & below);
            if (KIND == kNear) c.q_next.put(i, v[q]);
            else sp_list<KIND>(c)[i] = v[q];
        }
        at += __popc(m[q]);
    }
}

// Relax entries j[q] (those with ok[q]) of rows whose source distances are
// du[q]; every lane of the warp calls it.  Each step's accesses are issued for
// all kSpBatch entries before any answer is used: a small pass is a chain of
// round trips to L2, and this is four of them (columns and weights, distances,
// stamps, queue tails).  The stamp is taken without waiting for the minimum:
// whoever stamps v first queues it, and the distance in memory is then at most
// nd, its own or a smaller one.  (When the smaller one came in an earlier
// round the entry is spare; one per vertex and round at most, so the queues
// hold.)
__device__ __forceinline__ void sp_relax_batch(const SpCtx& c, const double* du, const int32_t* j, const bool* ok,
                                               SpFound& found, SpStage& g) {
    int32_t v[kSpBatch];
    double w[kSpBatch], cur[kSpBatch];
#pragma unroll
    for (int q = 0; q < kSpBatch; ++q) {
        v[q] = ok[q] ? c.col[j[q]] : 0;
        w[q] = ok[q] ? c.wt[j[q]] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kSpBatch; ++q) cur[q] = ok[q] ? sp_dist(c.dist, v[q]) : 0.0;
    int32_t old[kSpBatch], tag[kSpBatch];
#pragma unroll
    for (int q = 0; q < kSpBatch; ++q) {
        old[q] = tag[q] = 0;
        if (ok[q]) {
            ++found.exam;
            const double nd = du[q] + w[q];
            if (nd < cur[q]) {
                const unsigned long long nb = (unsigned long long)__double_as_longlong(nd);
                atomicMin(c.dist + v[q], nb);
                const bool near = nd < c.thr;
                // Rounds and phases start at 1 and 0; far tags are kept apart by their sign.
                tag[q] = near ? c.round : ~c.phase;
                old[q] = atomicExch((near ? c.near_stamp : c.far_stamp) + v[q], tag[q]);
                if (!near && nb < found.fmin) found.fmin = nb;
            }
        }
    }
    unsigned near_m[kSpBatch], far_m[kSpBatch];
    int32_t nnear = 0, nfar = 0;
#pragma unroll
    for (int q = 0; q < kSpBatch; ++q) {
        near_m[q] = __ballot_sync(0xffffffffu, old[q] != tag[q] && tag[q] > 0);
        far_m[q] = __ballot_sync(0xffffffffu, old[q] != tag[q] && tag[q] < 0);
        nnear += __popc(near_m[q]);
        nfar += __popc(far_m[q]);
    }
    if (nnear + nfar == 0) return;
    if (g.buf) {
        sp_append<kNear, kSpBatch>(c, g, near_m, v);
        sp_append<kFar, kSpBatch>(c, g, far_m, v);
        return;
    }
    const int lane = lane_id();
    int32_t base = 0;
    if (lane == 0 && nnear) base = c.q_base + atomicAdd(&c.slot->q_tail, nnear);
    if (lane == 1 && nfar) base = c.far_base + atomicAdd(&c.slot->far_add, nfar);
    int32_t near_at = __shfl_sync(0xffffffffu, base, 0), far_at = __shfl_sync(0xffffffffu, base, 1);
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int q = 0; q < kSpBatch; ++q) {
        if ((near_m[q] >> lane) & 1u) c.q_next.put(near_at + __popc(near_m[q] & below), v[q]);
        if ((far_m[q] >> lane) & 1u) c.far_cur[far_at + __popc(far_m[q] & below)] = v[q];
        near_at += __popc(near_m[q]);
        far_at += __popc(far_m[q]);
    }
}

// Relax [jb, je) of one row (distance du) with the whole warp.
__device__ __forceinline__ void sp_warp_range(const SpCtx& c, double du, int32_t jb, int32_t je, SpFound& found,
                                              SpStage& g) {
    for (int64_t j0 = jb; j0 < je; j0 += 32 * kSpBatch) {
        int32_t jj[kSpBatch];
        bool ok[kSpBatch];
        double dd[kSpBatch];
#pragma unroll
        for (int q = 0; q < kSpBatch; ++q) {
            const int64_t j = j0 + lane_id() + 32 * q;
            ok[q] = j < je;
            jj[q] = (int32_t)j;
            dd[q] = du;
        }
        sp_relax_batch(c, dd, jj, ok, found, g);
    }
}

// Relax [b, e) of the rows held by the warp's lanes (u < 0: none).  Rows
// longer than kSpDirect are appended, whole, to the chunk list of the CHUNK
// pass that follows.
__device__ __forceinline__ void sp_rows(const SpCtx& c, int32_t u, int32_t b, int32_t e, double du,
                                        SpFound& found, SpStage& g) {
    const int lane = lane_id();
    // Rows of a mesh: each lane its own, without votes and the scan below.
    const int32_t longest = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)(e - b));
    if (longest <= kSpBatch) {
        int32_t jj[kSpBatch];
        bool ok[kSpBatch];
        double dd[kSpBatch];
#pragma unroll
        for (int q = 0; q < kSpBatch; ++q) {
            jj[q] = b + q;
            ok[q] = q < e - b;
            dd[q] = du;
        }
        sp_relax_batch(c, dd, jj, ok, found, g);
        return;
    }
    if (longest > kSpDirect) {
        // One atomic for the warp's long rows; the first kOwn chunks of a row
        // are written by its lane, further ones by the warp.
        constexpr int32_t kOwn = 4;
        const int32_t nch = e - b > kSpDirect ? chunk_count(e - b, kSpChunk) : 0;
        int32_t incl = nch;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        int32_t pos = 0;
        if (lane == 31) pos = atomicAdd(&c.slot->c_tail, incl);
        pos = __shfl_sync(0xffffffffu, pos, 31) + incl - nch;
        for (int32_t k = 0; k < min(nch, kOwn); ++k) {
            const int32_t cb = b + k * kSpChunk;
            c.chunks[pos + k] = make_int4(u, cb, chunk_end(cb, kSpChunk, e), 0);
        }
        unsigned many = __ballot_sync(0xffffffffu, nch > kOwn);
        while (many) {
            const int leader = __ffs(many) - 1;
            many &= many - 1;
            const int32_t lu = __shfl_sync(0xffffffffu, u, leader), lb = __shfl_sync(0xffffffffu, b, leader);
            const int32_t lend = __shfl_sync(0xffffffffu, e, leader), lpos = __shfl_sync(0xffffffffu, pos, leader);
            const int32_t ln = __shfl_sync(0xffffffffu, nch, leader);
            for (int32_t k = kOwn + lane; k < ln; k += 32) {
                const int32_t cb = lb + k * kSpChunk;
                c.chunks[lpos + k] = make_int4(lu, cb, chunk_end(cb, kSpChunk, lend), 0);
            }
        }
        if (nch) e = b;
    }
    // Rows of 32 entries or more: the whole warp, one row at a time.
    unsigned med = longest >= 32 ? __ballot_sync(0xffffffffu, e - b >= 32) : 0u;
    while (med) {
        const int leader = __ffs(med) - 1;
        med &= med - 1;
        const int32_t lb = __shfl_sync(0xffffffffu, b, leader);
        const int32_t lend = __shfl_sync(0xffffffffu, e, leader);
        const double ld = __shfl_sync(0xffffffffu, du, leader);
        sp_warp_range(c, ld, lb, lend, found, g);
    }
    if (e - b >= 32) e = b;
    const int32_t d = e - b;
    // Shorter rows: gathered warp-wide over a scan of their lengths.
    int32_t incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    const int32_t excl = incl - d;
    const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
    for (int32_t k0 = 0; k0 < total; k0 += 32 * kSpBatch) {
        int32_t jj[kSpBatch];
        bool ok[kSpBatch];
        double dd[kSpBatch];
#pragma unroll
        for (int q = 0; q < kSpBatch; ++q) {
            const int32_t k = k0 + 32 * q + lane;
            int owner = 0;
#pragma unroll
            for (int s = 16; s >= 1; s >>= 1) {
                const int cand = owner + s;
                const int32_t ev = __shfl_sync(0xffffffffu, excl, cand);
                if (ev <= k) owner = cand;
            }
            const int32_t ob = __shfl_sync(0xffffffffu, b, owner);
            const int32_t oe = __shfl_sync(0xffffffffu, excl, owner);
            dd[q] = __shfl_sync(0xffffffffu, du, owner);
            ok[q] = k < total;
            jj[q] = ob + (k - oe);
        }
        sp_relax_batch(c, dd, jj, ok, found, g);
    }
}

__device__ __forceinline__ bool sp_barrier(SsspRunState* st, unsigned long long limit_ns, unsigned extra) {
    return grid_sync_leader(&st->bar_count, &st->bar_release, &st->status, NoLeader(), limit_ns, extra);
}

// Bucket-width adaptation: more LIGHT passes than this in a bucket halve
// the next bucket's width.
constexpr long long kSpAdaptLight = 4;

// End of the bucket that holds distance mn, on the grid thr + k * delta.
__device__ __forceinline__ double sp_next_thr(double thr, double delta, double mn) {
    double nthr = thr + delta;
    if (mn >= nthr) nthr = thr + delta * floor((mn - thr) / delta + 1.0);
    if (!(nthr > mn)) nthr = mn + delta;                // guards rounding
    if (!(nthr > mn)) nthr = nextafter(mn, INFINITY);  // delta below mn's ulp
    return nthr;
}

// The next pass, from the state and what the pass just finished appended.
__device__ __forceinline__ void sp_decide(SpState& s, const SpSlot& c) {
    const int32_t md0 = s.mode;
    ++s.passes;
    s.examined += c.examined;
    s.r_count += c.r_add;
    s.far_count += c.far_add;
    s.q_next += c.q_tail;
    if (c.fmin < s.fmin) s.fmin = c.fmin;
    if ((md0 == kLight || md0 == kHeavy) && c.c_tail > 0) {
        // Long rows were cut into chunks: a CHUNK pass finishes them in the
        // same round (same stamps, same next queue).
        s.nc = c.c_tail;
        s.chunk_of = md0;
        s.mode = kChunk;
        s.solo = s.nc <= kSoloChunks && s.solo_max > 0;
        return;
    }
    if (md0 == kChunk) ++s.chunk_passes;
    const int32_t md = md0 == kChunk ? s.chunk_of : md0;
    s.qsel ^= 1;
    s.nq = s.q_next;
    s.q_next = 0;
    s.nc = 0;
    if (md == kSplit) {
        s.thr = s.new_thr;
        ++s.splits;
    } else if (md == kHeavy) {
        s.r_count = 0;
        ++s.epoch;
        ++s.heavy_passes;
    } else {
        ++s.light_passes;
    }
    int32_t next = kDone;
    int32_t solo_max = s.solo_max;
    if (s.nq > 0) {
        next = kLight;
    } else if (md == kLight && s.r_count > 0) {
        next = kHeavy;
        s.nq = s.r_count;
    } else if (s.far_count > 0) {
        // Next bucket: the one holding the smallest pending far distance (its
        // recorded minimum can be low when an entry settled later; a SPLIT
        // that queues nothing then repeats with the exact minimum of the
        // entries it kept).
        //
        // Its width: halved after a bucket that took more than kSpAdaptLight
        // LIGHT passes (its vertices were relaxed again and again), doubled
        // after one that took at most two and examined little (passes with
        // too little work for the grid).  Exact distances do not depend on
        // it: the passes form a label-correcting loop in which a HEAVY pass
        // that lowers a distance inside the bucket sends it back to a LIGHT
        // pass, and R is refilled after every HEAVY pass.
        const long long lp = s.light_passes - s.lp_mark;
        const unsigned long long ex = s.examined - s.ex_mark;
        if (lp > kSpAdaptLight) s.width = fmax(s.width * 0.5, s.width_min);
        else if (lp <= 2 && ex < s.adapt_work) s.width = fmin(s.width * 2.0, s.width_max);
        s.lp_mark = s.light_passes;
        s.ex_mark = s.examined;
        const double mn = s.fmin == ~0ull ? s.thr : __longlong_as_double((long long)s.fmin);
        s.new_thr = sp_next_thr(s.thr, s.width, mn);
        s.fmin = ~0ull;
        s.nq = s.far_count;
        s.far_count = 0;
        s.fsel ^= 1;
        ++s.phase;
        next = kSplit;
        solo_max *= 4;  // one distance per entry, no row
    }
    ++s.round;
    // Budgets: a correct run needs far fewer passes and far less time; past
    // either, stop with an error status.
    if (next != kDone && (s.passes > s.pass_budget || c.stop)) {
        s.failed = 1;
        next = kDone;
    }
    s.mode = next;
    s.solo = next != kDone && s.nq <= solo_max;
}

}  // namespace

// A warp's findings into its block's totals.
__device__ __forceinline__ void sp_total(const SpFound& found, unsigned long long* examined,
                                         unsigned long long* fmin) {
    const unsigned exam = __reduce_add_sync(0xffffffffu, found.exam);
    if (lane_id() == 0 && exam) atomicAdd(examined, (unsigned long long)exam);
    if (__any_sync(0xffffffffu, found.fmin != ~0ull)) {
        unsigned long long m = found.fmin;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane_id() == 0) atomicMin(fmin, m);
    }
}

// One pass's share of warp `warp` of `nwarps` (thread `tid` of `nt`).
__device__ __forceinline__ void sp_pass(const SpState& s, SpCtx& c, const SpQueue& q_cur, int32_t* fa, int32_t* fb,
                                        int64_t tid, int64_t nt, SpFound& found,
                                        SpStage& g) {
    const int lane = lane_id();
    const int64_t warp = tid >> 5, nwarps = nt >> 5;
    const bool split = c.le != nullptr;
    if (s.mode == kChunk) {
        // The long rows of the pass just finished, a chunk per warp.
        for (int64_t i = warp; i < s.nc; i += nwarps) {
            const int4 ch = __ldcg(c.chunks + i);
            const double du = sp_dist(c.dist, ch.x);
            sp_warp_range(c, du, ch.y, ch.z, found, g);
        }
    } else if (s.mode == kSplit) {
        const int32_t* far = s.fsel ? fa : fb;
        const double old_thr = s.thr, nthr = s.new_thr;
        for (int64_t i = tid; i - lane < s.nq; i += nt) {
            int32_t v = 0;
            bool near = false, keep = false;
            if (i < s.nq) {
                v = __ldcg(far + i);
                const double d = sp_dist(c.dist, v);
                // Below old_thr it was settled in an earlier bucket.
                if (d >= old_thr && d < nthr) {
                    near = atomicExch(c.near_stamp + v, c.round) != c.round;
                } else if (d >= old_thr) {
                    keep = atomicExch(c.far_stamp + v, ~c.phase) != ~c.phase;
                    const unsigned long long db = (unsigned long long)__double_as_longlong(d);
                    if (db < found.fmin) found.fmin = db;
                }
            }
            const unsigned near_m = __ballot_sync(0xffffffffu, near), keep_m = __ballot_sync(0xffffffffu, keep);
            sp_append<kNear, 1>(c, g, &near_m, &v);
            sp_append<kFar, 1>(c, g, &keep_m, &v);
        }
    } else {
        // Queue rows, 32 per warp; on small queues fewer, so that their rows
        // spread over every warp instead of queueing behind each other.
        int64_t per = 32;
        while (per > 1 && nwarps * (per >> 1) >= s.nq) per >>= 1;
        for (int64_t base = warp * per; base < s.nq; base += nwarps * per) {
            const int64_t i = base + lane;
            int32_t u = -1, b = 0, e = 0;
            double du = 0.0;
            bool settled = false;  // joins R
            if (lane < per && i < s.nq) {
                if (s.mode == kLight) {
                    u = q_cur.get((int32_t)i);
                    b = c.rp[u];
                    e = split ? c.le[u] : c.rp[u + 1];
                    du = sp_dist(c.dist, u);
                    if (split) settled = atomicExch(c.r_stamp + u, c.epoch) != c.epoch;
                } else {
                    u = __ldcg(c.R + i);
                    b = c.le[u];
                    e = c.rp[u + 1];
                    du = sp_dist(c.dist, u);
                }
            }
            sp_rows(c, u, b, e, du, found, g);
            if (split && s.mode == kLight) {
                const unsigned settled_m = __ballot_sync(0xffffffffu, settled);
                sp_append<kSettled, 1>(c, g, &settled_m, &u);
            }
        }
    }
}

__global__ void __launch_bounds__(kSsspThreads, 2) sssp_persistent_kernel(
    int32_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ le, const int32_t* __restrict__ col,
    const double* __restrict__ wt, int32_t src, double inf, double* dist_d, int32_t* qa, int32_t* qb, int4* chunks,
    int32_t* fa, int32_t* fb, int32_t* near_stamp, int32_t* far_stamp, int32_t* r_stamp, int32_t* R,
    SsspRunState* st, const int32_t* __restrict__ perm, double* out) {
    unsigned long long* dist = reinterpret_cast<unsigned long long*>(dist_d);
    const int64_t gtid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t gsize = (int64_t)gridDim.x * blockDim.x;
    const bool split = le != nullptr;
    __shared__ SpState s;
    __shared__ SpSlot own;  // the slot of a solo pass
    __shared__ unsigned long long s_fmin, s_exam, s_t0;
    // Solo runs: the two near queues' first entries.  Grid passes: the warps'
    // staged vertices, and how many are left at the end, then where they go.
    __shared__ int32_t s_lists[kSpWarps * kSpKinds * kSpStage];
    static_assert(kSpWarps * kSpKinds * kSpStage >= 2 * kSoloQueue, "the solo queues fit");
    auto fast = [&](int32_t sel) { return s_lists + sel * kSoloQueue; };
    __shared__ int32_t s_left[kSpKinds][kSpWarps];
    const unsigned long long limit_ns = st->bar_limit_ns;
    const unsigned extra = st->bar_extra;

    // ---- init
    if (perm) src = perm[src];
    const unsigned long long ib = (unsigned long long)__double_as_longlong(inf);
    for (int64_t v = gtid; v < n; v += gsize) {
        dist[v] = (v == src) ? 0ull : ib;
        near_stamp[v] = -1;
        far_stamp[v] = 0;
        if (split) r_stamp[v] = -1;
    }
    if (threadIdx.x == 0) {
        s = st->s;
        s_fmin = ~0ull;
        s_exam = 0;
        s_t0 = global_timer_ns();
    }
    if (gtid == 0) {
        qa[0] = src;
        for (int k = 0; k < 3; ++k) st->slot[k].fmin = ~0ull;
    }
    if (!sp_barrier(st, limit_ns, extra)) return;

    SpCtx c;
    c.rp = rp;
    c.le = le;
    c.col = col;
    c.wt = wt;
    c.dist = dist;
    c.near_stamp = near_stamp;
    c.far_stamp = far_stamp;
    c.r_stamp = r_stamp;
    c.R = R;
    c.chunks = chunks;
    unsigned turn = 0;  // the grid's passes: which slot is filled
    while (s.mode != kDone) {
        auto context = [&](int32_t cap) {
            c.q_next = SpQueue{fast(s.qsel ^ 1), s.qsel ? qa : qb, cap};
            c.far_cur = s.fsel ? fb : fa;
            c.thr = s.thr;
            c.round = s.round;
            c.phase = s.phase;
            c.epoch = s.epoch;
            c.q_base = s.q_next;
            c.r_base = s.r_count;
            c.far_base = s.far_count;
        };
        if (s.solo) {
            // ---- a run of small passes on block 0, the others at the barrier
            // below: a pass then costs its own chain of loads and a block
            // barrier, not a grid barrier and a state read through L2.
            if (blockIdx.x == 0) {
                // The queue's first entries move to shared memory for the run.
                const int32_t held = s.mode == kLight ? min(s.nq, kSoloQueue) : 0;
                for (int32_t i = threadIdx.x; i < held; i += blockDim.x)
                    fast(s.qsel)[i] = __ldcg((s.qsel ? qb : qa) + i);
                // Entries that an unfinished round (its chunks come next) has
                // queued move as well.
                const int32_t held_next = min(s.q_next, kSoloQueue);
                for (int32_t i = threadIdx.x; i < held_next; i += blockDim.x)
                    fast(s.qsel ^ 1)[i] = __ldcg((s.qsel ? qa : qb) + i);
                const unsigned long long t_run = global_timer_ns();
                if (threadIdx.x == 0) {
                    own.q_tail = own.c_tail = own.r_add = own.far_add = own.stop = 0;
                    own.fmin = ~0ull;
                    own.examined = 0;
                }
                __syncthreads();
                c.slot = &own;
                for (int turns = 0; s.solo && turns < kSoloTurns; ++turns) {
                    context(kSoloQueue);
                    const SpQueue q_cur{fast(s.qsel), s.qsel ? qb : qa, kSoloQueue};
                    SpFound found;
                    SpStage stage{nullptr, {0, 0, 0}};
                    sp_pass(s, c, q_cur, fa, fb, threadIdx.x, blockDim.x, found, stage);
                    sp_total(found, &own.examined, &own.fmin);
                    __syncthreads();
                    if (threadIdx.x == 0) {
                        const bool look = solo_look(turns, limit_ns);
                        const unsigned long long now = look ? global_timer_ns() : 0;
                        own.stop = look && now - s_t0 > kSsspTimeBudgetNs;
                        sp_decide(s, own);
                        own.q_tail = own.c_tail = own.r_add = own.far_add = 0;
                        own.fmin = ~0ull;
                        own.examined = 0;
                        // The others' wait is bounded: hand back well before it ends.
                        if (look && now - t_run > limit_ns / 8) s.solo = 0;
                    }
                    __syncthreads();
                }
                // Back to global memory: the queue that the next pass reads,
                // and the one that an unfinished round fills.
                const int32_t back = s.mode == kLight ? min(s.nq, kSoloQueue) : 0;
                for (int32_t i = threadIdx.x; i < back; i += blockDim.x)
                    (s.qsel ? qb : qa)[i] = fast(s.qsel)[i];
                const int32_t back_next = min(s.q_next, kSoloQueue);
                for (int32_t i = threadIdx.x; i < back_next; i += blockDim.x)
                    (s.qsel ? qa : qb)[i] = fast(s.qsel ^ 1)[i];
                // One pass of the whole grid follows even where the next is
                // small: the run above ended by its own limits then.
                if (threadIdx.x == 0) {
                    s.solo = 0;
                    st->s = s;
                }
            }
            if (!sp_barrier(st, limit_ns, extra)) return;
            if (blockIdx.x != 0 && threadIdx.x < sizeof(SpState) / 4)
                reinterpret_cast<int32_t*>(&s)[threadIdx.x] =
                    __ldcg(reinterpret_cast<const int32_t*>(&st->s) + threadIdx.x);
            __syncthreads();
            continue;
        }
        SpSlot* slot = &st->slot[turn % 3];
        context(0);
        c.slot = slot;
        const SpQueue q_cur{nullptr, s.qsel ? qb : qa, 0};
        SpFound found;
        const int wid = threadIdx.x >> 5, lane = lane_id();
        SpStage stage{s_lists + wid * kSpKinds * kSpStage, {0, 0, 0}};
        sp_pass(s, c, q_cur, fa, fb, gtid, gsize, found, stage);
        // What the warps have left and the block's totals, then the barrier.
        if (lane < kSpKinds) s_left[lane][wid] = lane == kNear ? stage.n[kNear] : lane == kFar ? stage.n[kFar] : stage.n[kSettled];
        sp_total(found, &s_exam, &s_fmin);
        __syncthreads();
        if (wid == 0) {
            // Lane k takes kind k's places for the whole block.
            int32_t excl[kSpKinds], take = 0;
#pragma unroll
            for (int k = 0; k < kSpKinds; ++k) {
                const int32_t x = lane < kSpWarps ? s_left[k][lane] : 0;
                int32_t incl = x;
#pragma unroll
                for (int o = 1; o < kSpWarps; o <<= 1) {
                    const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                excl[k] = incl - x;
                const int32_t total = __shfl_sync(0xffffffffu, incl, kSpWarps - 1);
                if (lane == k) take = total;
            }
            int32_t at = 0;
            if (take) {
                if (lane == kNear) at = sp_base<kNear>(c) + atomicAdd(sp_tail<kNear>(c), take);
                else if (lane == kFar) at = sp_base<kFar>(c) + atomicAdd(sp_tail<kFar>(c), take);
                else at = sp_base<kSettled>(c) + atomicAdd(sp_tail<kSettled>(c), take);
            }
#pragma unroll
            for (int k = 0; k < kSpKinds; ++k) {
                const int32_t to = __shfl_sync(0xffffffffu, at, k);
                if (lane < kSpWarps) s_left[k][lane] = to + excl[k];
            }
        } else if (threadIdx.x == 32) {
            if (s_exam) atomicAdd(&slot->examined, s_exam);
            if (s_fmin != ~0ull) atomicMin(&slot->fmin, s_fmin);
            s_exam = 0;
            s_fmin = ~0ull;
            if (blockIdx.x == 0) {
                SpSlot* clear = &st->slot[(turn + 1) % 3];
                clear->q_tail = clear->c_tail = clear->r_add = clear->far_add = clear->stop = 0;
                clear->fmin = ~0ull;
                clear->examined = 0;
                if (global_timer_ns() - s_t0 > kSsspTimeBudgetNs) slot->stop = 1;
            }
        }
        __syncthreads();
        sp_write<kNear>(c, stage, s_left[kNear][wid]);
        sp_write<kFar>(c, stage, s_left[kFar][wid]);
        sp_write<kSettled>(c, stage, s_left[kSettled][wid]);
        if (!sp_barrier(st, limit_ns, extra)) return;
        if (threadIdx.x == 0) {
            SpSlot f;
            f.q_tail = __ldcg(&slot->q_tail);
            f.c_tail = __ldcg(&slot->c_tail);
            f.r_add = __ldcg(&slot->r_add);
            f.far_add = __ldcg(&slot->far_add);
            f.fmin = __ldcg(&slot->fmin);
            f.examined = __ldcg(&slot->examined);
            f.stop = __ldcg(&slot->stop);
            sp_decide(s, f);
        }
        ++turn;
        __syncthreads();
    }
    if (gtid == 0) {
        st->s = s;
        if (s.failed) st->status = kDevOverflow;
    }

    // ---- results in the caller's ids
    if (perm) {
        for (int64_t v = gtid; v < n; v += gsize) out[v] = sp_dist(dist, perm[v]);
    }
}

// ------------------------------------------------------------------- host
namespace {

__global__ void sp_light_end_kernel(int32_t n, const int32_t* __restrict__ rp, const double* __restrict__ sw_w,
                                    double delta, int32_t* light_end) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x) {
        int32_t lo = rp[u], hi = rp[u + 1];
        while (lo < hi) {
            const int32_t mid = row_middle(lo, hi);
            if (sw_w[mid] < delta) lo = mid + 1;
            else hi = mid;
        }
        light_end[u] = lo;
    }
}

__global__ void sp_reached_kernel(int32_t n, const int32_t* __restrict__ rp, const double* __restrict__ dist,
                                  double inf, unsigned long long* out) {
    unsigned long long e = 0, r = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        if (dist[v] != inf) {
            e += (unsigned long long)(rp[v + 1] - rp[v]);
            ++r;
        }
    }
    e = warp_sum(e);
    r = warp_sum(r);
    if (lane_id() == 0) {
        atomicAdd(out, e);
        atomicAdd(out + 1, r);
    }
}

}  // namespace

bool sssp_persistent_available(ghb_workspace* ws, int* blocks) {
    static int cached[64] = {0};
    static bool known[64] = {false};
    const int dev = ws->device;
    if (dev < 0 || dev >= 64) return false;
    if (!known[dev]) {
        int coop = 0, per_sm = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        if (coop && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sssp_persistent_kernel, kSsspThreads, 0) ==
                        cudaSuccess)
            cached[dev] = std::min(per_sm, 2) * ws->num_sms;
        known[dev] = true;
    }
    *blocks = cached[dev];
    return cached[dev] > 0;
}

// Light ends of a resident graph's weight-sorted rows for width delta,
// cached on the handle until a call asks for another width.
int graph_light_ends(ghb_workspace* ws, ghb_graph* g, double delta, const int32_t** le) {
    if (!g->sw_le) {
        GHB_CUDA_TRY(cudaMalloc(&g->sw_le, sizeof(int32_t) * (size_t)g->n));
        g->device_bytes += 4 * (int64_t)g->n;
        g->sw_le_delta = -1.0;
    }
    if (g->sw_le_delta != delta) {
        GHB_TRY(launch(ws, sp_light_end_kernel, dim3(grid_for(g->n, 256, ws->num_sms * 8)), dim3(256), 0, g->n,
                       (const int32_t*)g->rowptr, (const double*)g->sw_w, delta, g->sw_le));
        g->sw_le_delta = delta;
    }
    *le = g->sw_le;
    return GHB_OK;
}

// One cooperative launch for the whole traversal.  rp/col/wt: the rows to
// relax (a resident graph's weight-sorted copy when le is given, whose
// light ranges [rp[u], le[u]) hold the entries below delta).  dist: per
// vertex in the graph's ids; with perm, src is the caller's id and
// out[v] = dist[perm[v]] as well.  m: the rows' entries where the caller
// knows them, else -1.
int sssp_persistent_run(ghb_workspace* ws, int32_t n, const int32_t* rp, const int32_t* le, const int32_t* col,
                        const double* wt, int64_t m, int32_t src, double inf, double delta, double* dist,
                        const int32_t* perm, double* out, ghb_traversal_stats* stats) {
    int blocks = 0;
    if (!sssp_persistent_available(ws, &blocks)) {
        set_error("cooperative launch unavailable");
        return GHB_ERR_UNSUPPORTED;
    }
    cudaStream_t st = ws->stream;
    if (m < 0) {
        int32_t* hp = reinterpret_cast<int32_t*>(ws->host_pinned);
        GHB_CUDA_TRY(cudaMemcpyAsync(hp, rp + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
        GHB_CUDA_TRY(cudaStreamSynchronize(st));
        m = hp[0];
    }
    // Chunks of one pass: rows over kSpDirect entries, ceil(len / kSpChunk)
    // each, so fewer than m / kSpChunk + m / kSpDirect.
    const int64_t chunk_cap = m / 32 + 64;
    auto carve = [&](Carver& c, int32_t** qa, int32_t** qb, int4** ch, int32_t** fa, int32_t** fb,
                     int32_t** ns, int32_t** fs, int32_t** rs, int32_t** R, SsspRunState** rs_state) {
        *qa = c.take<int32_t>(n);
        *qb = c.take<int32_t>(n);
        *ch = c.take<int4>(chunk_cap);
        *fa = c.take<int32_t>(n);
        *fb = c.take<int32_t>(n);
        *ns = c.take<int32_t>(n);
        *fs = c.take<int32_t>(n);
        *rs = c.take<int32_t>(le ? n : 1);
        *R = c.take<int32_t>(le ? n : 1);
        *rs_state = c.take<SsspRunState>(1);
    };
    int32_t *qa, *qb, *fa, *fb, *ns, *fs, *rs, *R;
    int4* ch;
    SsspRunState* rstate;
    Carver sizing(nullptr);
    carve(sizing, &qa, &qb, &ch, &fa, &fb, &ns, &fs, &rs, &R, &rstate);
    GHB_TRY(ws_reserve(ws, sizing.off));
    Carver c(ws->scratch);
    carve(c, &qa, &qb, &ch, &fa, &fb, &ns, &fs, &rs, &R, &rstate);

    // The start state (pageable source: staged by the copy).
    SsspRunState start;
    SsspRunState* h0 = &start;
    std::memset(static_cast<void*>(h0), 0, sizeof(SsspRunState));
    h0->bar_limit_ns = (unsigned long long)ws->tune.barrier_limit_us * 1000ull;
    h0->bar_extra = (unsigned)ws->tune.barrier_extra;
    h0->s.mode = kLight;
    h0->s.round = 1;
    h0->s.nq = 1;
    h0->s.fmin = ~0ull;
    h0->s.thr = delta;
    // Every productive pass lowers some distance: 64 passes per vertex bound
    // any correct run, as in the host-driven loop.
    h0->s.pass_budget = 64ll * n + 1024;
    // Bucket widths: delta, or from delta / 64 to delta * 64 when they adapt;
    // a bucket is small below eight entries per thread.
    const bool adapt = ws->tune.sssp_adapt != 0;
    h0->s.width = delta;
    h0->s.width_min = adapt ? delta / 64.0 : delta;
    h0->s.width_max = adapt ? delta * 64.0 : delta;
    h0->s.adapt_work = 8ull * (unsigned long long)blocks * kSsspThreads;
    // Small passes: a few entries per thread of one block.
    h0->s.solo_max = (int32_t)std::min<int64_t>(kSoloQueue, std::max<int64_t>(16, kSoloEntries * (int64_t)n / std::max<int64_t>(m, 1)));
    h0->s.solo = 1;
    GHB_CUDA_TRY(cudaMemcpyAsync(rstate, h0, sizeof(SsspRunState), cudaMemcpyHostToDevice, st));
    if (stats) GHB_CUDA_TRY(cudaEventRecord(ws->ev_start, st));
    GHB_TRY(launch_coop(ws, sssp_persistent_kernel, dim3(blocks), dim3(kSsspThreads), 0, n, rp, le, col, wt, src, inf,
                        dist, qa, qb, ch, fa, fb, ns, fs, rs, R, rstate, perm, out));
    if (stats) GHB_CUDA_TRY(cudaEventRecord(ws->ev_stop, st));
    // The reached vertices and their entries, counted behind the traversal:
    // one wait for both.
    constexpr size_t kReachedWord = (sizeof(SsspRunState) + 7) / 8;
    static_assert(kReachedWord + 2 <= (size_t)kHostPinnedWords, "the run state and two sums fit the pinned words");
    if (stats) {
        unsigned long long* acc = reinterpret_cast<unsigned long long*>(ws->dev_small);
        GHB_CUDA_TRY(cudaMemsetAsync(acc, 0, 2 * sizeof(unsigned long long), st));
        GHB_TRY(launch(ws, sp_reached_kernel, dim3(grid_for(n, 256, ws->num_sms * 8)), dim3(256), 0, n, rp,
                       (const double*)dist, inf, acc));
        GHB_CUDA_TRY(cudaMemcpyAsync(ws->host_pinned + kReachedWord, acc, 2 * sizeof(unsigned long long),
                                     cudaMemcpyDeviceToHost, st));
    }
    GHB_CUDA_TRY(cudaMemcpyAsync(ws->host_pinned, rstate, sizeof(SsspRunState), cudaMemcpyDeviceToHost, st));
    GHB_CUDA_TRY(cudaStreamSynchronize(st));
    SsspRunState h;
    std::memcpy(&h, ws->host_pinned, sizeof(h));
    if (h.status == kDevOverflow) {
        set_error("SSSP: pass or time budget exhausted");
        return GHB_ERR_LIMIT;
    }
    if (h.status != kDevOk) {
        set_error("SSSP: grid barrier timed out");
        return GHB_ERR_TIMEOUT;
    }
    if (stats) {
        float ms = 0.f;
        GHB_CUDA_TRY(cudaEventElapsedTime(&ms, ws->ev_start, ws->ev_stop));
        const int64_t* ha = ws->host_pinned + kReachedWord;
        stats->levels = (int32_t)(h.s.light_passes + h.s.heavy_passes + h.s.chunk_passes);
        stats->pull_levels = (int32_t)h.s.splits;
        stats->edges_reached = (int64_t)ha[0];
        stats->reached = (int64_t)ha[1];
        stats->edges_examined = (int64_t)h.s.examined;
        stats->device_ms = ms;
    }
    return GHB_OK;
}

}  // namespace ghb
