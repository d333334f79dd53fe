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

}  // namespace culsh_b200
