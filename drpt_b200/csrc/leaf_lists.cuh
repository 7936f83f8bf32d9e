// The per-point candidate lists that the whole-leaf kernels write.
#pragma once

#include "common.cuh"

namespace drpt {

// A block's `rows` points get empty lists: what a tile of a leaf beyond the kernel's
// limit leaves.  The build then ends with an error, but its fold and re-rank run
// before the host sees it, and the re-rank reads the rows that the lists name.
template <int KP>
__device__ __forceinline__ void empty_lists(const int32_t *points, int rows, int32_t *idx,
                                            float *dist) {
  for (int e = threadIdx.x; e < rows * KP; e += blockDim.x) {
    const int64_t o = (int64_t)points[e / KP] * KP + e % KP;
    idx[o] = -1;
    dist[o] = __int_as_float(0x7f800000);
  }
}

}  // namespace drpt
