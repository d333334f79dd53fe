// Index arithmetic that has to stay inside 64 (or unsigned 32) bits at the largest sizes the engine takes.
// Plain C++ as well as CUDA.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CULSH_HD __host__ __device__ __forceinline__
#else
#define CULSH_HD inline
#endif

namespace culsh_b200 {

// First unit of a CTA's tile of `per_tile` units inside its table.  A table of 2^29 rows with keys of
// sixteen words has 2^31 quarters of a key.
CULSH_HD int64_t tile_first(uint32_t tile, int per_tile) { return (int64_t)tile * per_tile; }

// f(row) for the rows first, first + stride, ... below n.  Unsigned: the step past the last row may pass 2^31.
template <typename F>
CULSH_HD void walk_rows(uint32_t first, uint32_t stride, int n, F&& f) {
    for (uint32_t row = first; row < (uint32_t)n; row += stride) f((int)row);
}

// Blocks of `per` rows in n.  Unsigned: n + per - 1 may pass 2^31.
CULSH_HD int row_blocks(int n, int per) { return (int)(((uint32_t)n + (uint32_t)per - 1u) / (uint32_t)per); }

}  // namespace culsh_b200
