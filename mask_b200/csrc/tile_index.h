// Where the ids of a tile begin.  Tiles are numbered with 32 bits, their ids are not: a group may hold every tile of a
// matrix (groups of 2^28 tiles and more can be asked for, and so can one group for a window of that many), and 2^28 tiles are 2^31 ids.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MASK_BOTH_SIDES __host__ __device__ __forceinline__
#else
#define MASK_BOTH_SIDES inline
#endif

namespace mask {

MASK_BOTH_SIDES constexpr int64_t ids_before_tile(uint32_t tile) { return (int64_t)tile * 8; }

}  // namespace mask
