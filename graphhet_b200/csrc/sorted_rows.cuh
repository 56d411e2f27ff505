// Rows from sorted keys (row << bits) | col: shared by the CSR builder and the
// relabelling.
#pragma once

#include "common.cuh"

namespace ghb {

// rowptr[r] = at for r in [r0, r1].  Most gaps between neighbouring entries
// hold a row or two; a long one (a stretch of isolated vertices: nearly half
// of an RMAT graph's ids end up behind the last entry of its relabelled rows)
// is left in the block's list, which all of its threads then fill.  (One
// thread filling the 1.8 M tail rows of an RMAT-22 graph took 6.4 ms.)
struct RowGaps {
    static constexpr int kLong = 64, kCap = 64;
    int32_t count;
    int32_t r0[kCap], r1[kCap], at[kCap];
};
__device__ __forceinline__ void fill_rows(RowGaps& g, int32_t* rowptr, int64_t r0, int64_t r1, int32_t at) {
    if (r1 - r0 >= RowGaps::kLong) {
        const int i = atomicAdd(&g.count, 1);
        if (i < RowGaps::kCap) {
            g.r0[i] = (int32_t)r0;
            g.r1[i] = (int32_t)r1;
            g.at[i] = at;
            return;
        }
    }
    for (int64_t r = r0; r <= r1; ++r) rowptr[r] = at;
}
// Every thread of the block, once, after a barrier that follows its fill_rows
// calls.  The list is not emptied: a kernel that fills twice sets count to zero
// between two barriers.
__device__ __forceinline__ void fill_long_rows(RowGaps& g, int32_t* rowptr) {
    const int n = min(g.count, RowGaps::kCap);
    for (int i = 0; i < n; ++i)
        for (int64_t r = (int64_t)g.r0[i] + threadIdx.x; r <= g.r1[i]; r += blockDim.x) rowptr[r] = g.at[i];
}

}  // namespace ghb
