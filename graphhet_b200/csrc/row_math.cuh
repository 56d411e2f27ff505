// Positions in a CSR of up to 2^31 - 1 entries, in 32 bits: sums that pass 2^31
// (a chunk's end, a rounded length) are taken unsigned.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define GHB_HD __host__ __device__ __forceinline__
#else
#define GHB_HD inline
#endif

namespace ghb {

// Chunks of `size` entries that hold `len` entries.
GHB_HD int32_t chunk_count(int32_t len, int32_t size) {
    return (int32_t)(((uint32_t)len + (uint32_t)size - 1u) / (uint32_t)size);
}

// End of the chunk that begins at `at` in a row that ends at `end`.
GHB_HD int32_t chunk_end(int32_t at, int32_t size, int32_t end) {
    const uint32_t e = (uint32_t)at + (uint32_t)size;
    return e < (uint32_t)end ? (int32_t)e : end;
}

// Middle of positions lo <= hi (their sum passes 2^31 from 2^30 entries on).
GHB_HD int32_t row_middle(int32_t lo, int32_t hi) { return lo + ((hi - lo) >> 1); }

}  // namespace ghb
