// A warp's sorted list of up to 32 (distance, id) pairs, one per lane, in
// ascending (distance, id) order (ids compared as unsigned, so that an empty
// entry, +inf and -1, comes last).
#pragma once

#include "common.cuh"

namespace drpt {

__device__ __forceinline__ bool qbefore(float da, int32_t ia, float db, int32_t ib) {
  return da < db || (da == db && (uint32_t)ia < (uint32_t)ib);
}

// Bitonic sort of 32 (d, id) pairs held one per lane, ascending.
__device__ __forceinline__ void warp_sort32(float &d, int32_t &id, int lane) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const float od = __shfl_xor_sync(kFull, d, stride);
      const int32_t oi = __shfl_xor_sync(kFull, id, stride);
      const bool up = (lane & size) == 0 || size == 32;
      const bool lower = (lane & stride) == 0;
      const bool mine_first = qbefore(d, id, od, oi);
      const bool keep = (lower == up) ? mine_first : !mine_first;
      if (!keep) {
        d = od;
        id = oi;
      }
    }
}

// L (sorted over the lanes) <- the 32 smallest of L and a sorted batch: the
// minimum of L and the reversed batch is bitonic; a bitonic clean sorts it.
__device__ __forceinline__ void warp_merge32(float &ld, int32_t &li, float d, int32_t id,
                                             int lane) {
  const float rd = __shfl_sync(kFull, d, 31 - lane);
  const int32_t ri = __shfl_sync(kFull, id, 31 - lane);
  if (qbefore(rd, ri, ld, li)) {
    ld = rd;
    li = ri;
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    const float od = __shfl_xor_sync(kFull, ld, stride);
    const int32_t oi = __shfl_xor_sync(kFull, li, stride);
    const bool lower = (lane & stride) == 0;
    const bool mine_first = qbefore(ld, li, od, oi);
    if (lower != mine_first) {
      ld = od;
      li = oi;
    }
  }
}

// The warp's sorted list <- its 32 smallest with this lane's candidate
// (id < 0: none).  Only candidates before the list's k-th entry enter; a few
// are inserted one by one (a ballot and a shift each), more are sorted and
// merged as a batch.  Every lane takes part in every shuffle.
__device__ __forceinline__ void warp_take(float &ld, int32_t &li, float d, int32_t id, int k,
                                          int lane) {
  const float kd = __shfl_sync(kFull, ld, k - 1);
  const int32_t ki = __shfl_sync(kFull, li, k - 1);
  const bool pass = id >= 0 && qbefore(d, id, kd, ki);
  unsigned m = __ballot_sync(kFull, pass);
  if (m == 0) return;
  if (__popc(m) > 5) {
    float bd = pass ? d : __int_as_float(0x7f800000);
    int32_t bi = pass ? id : -1;
    warp_sort32(bd, bi, lane);
    warp_merge32(ld, li, bd, bi, lane);
    return;
  }
  do {
    const int src = __ffs(m) - 1;
    m &= m - 1;
    const float v = __shfl_sync(kFull, d, src);
    const int32_t i = __shfl_sync(kFull, id, src);
    const int at = __popc(__ballot_sync(kFull, qbefore(ld, li, v, i)));
    const float ud = __shfl_up_sync(kFull, ld, 1);
    const int32_t ui = __shfl_up_sync(kFull, li, 1);
    if (lane == at) {
      ld = v;
      li = i;
    } else if (lane > at) {
      ld = ud;
      li = ui;
    }
  } while (m);
}

}  // namespace drpt
