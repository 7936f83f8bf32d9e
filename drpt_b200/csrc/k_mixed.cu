// Mixed-precision form of the leaf brute force.
//
// The reference scores every leaf row exactly in FP32 (mdrpt.cpp:123-212).
// The mixed form keeps its global trees (projection + histogram-median
// splits) but brute-forces each whole global leaf with BF16 Gram tiles on the
// tensor cores and wins the accuracy back afterwards:
//
//   K8  k_leaf_index    per tree and point: its row in the tree's leaf order
//                       and its leaf
//       k_leaf_mean     per tree and global leaf: the mean of its first rows
//       k_leaf_stage    per point, read once in index order, for every tree of
//                       a chunk: subtract its leaf's mean (FP32), round to
//                       BF16, store at its row in that tree's leaf order, norm
//                       of the rounded row
//   K9  k_tile_plan     row tiles of 128 points of every leaf
//   K10 k_leaf_mma      per row tile: TMA-fed tcgen05 MMAs (BF16 x BF16 ->
//                       FP32 in Tensor Memory, M = 128 rows, N = 64 to 256
//                       columns per tile, K = the padded dimension), epilogue
//                       scores ||y||^2 - 2 x.y per column and keeps each
//                       row's KP best in registers (threshold filter seeded
//                       from the running list, per-thread shared-memory
//                       buffer, sort + merge networks); k_fold_lists then
//                       folds them into the point's running list of the KP
//                       best distinct candidates over the trees built so far
//   K11 k_rerank        per point: the running list's KP candidates rescored with the
//                       exact sequential FP32 distance of the plain form, the
//                       k best kept; candidates whose FP32 distance lies within
//                       a relative 2^-16 of the k-th are re-ordered by an FP64
//                       distance
//
// Centring on the leaf mean keeps the BF16 rounding error of x.y small next
// to the squared distances that are ranked (values of a few tens instead of a
// few hundreds for the synthetic workloads).
#include <cuda.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "leaf_lists.cuh"
#include "sm100.cuh"

namespace drpt {
namespace {

using namespace sm100;

constexpr int kTM = 128;            // rows per tile (M)
// Four shapes of the leaf kernel, by how many 128-byte K blocks a row has.
// In all of them the 128 rows of a tile (A) meet the leaf's columns in tiles
// of `tn` (B) through a ring of stages of one K block each, into two
// accumulators.
//   0: kb <= 2, A resident, 64 columns, 3 CTAs per SM (32 keys per row: 2).
//      The epilogue bounds it, so the warps per SM count.
//   1: kb <= 4 and 16 keys, A resident (64 KB), 64 columns, 2 CTAs per SM.
//   2: a stage holds a K block of A too, 128 columns, 2 CTAs per SM.
//   3: as 2 with 256 columns, 1 CTA per SM (wide rows, or fairly wide rows and
//      large leaves: wide_rows).
// Past shape 0 the feed from L2 bounds the kernel (64-column tiles with A
// streamed took in 48 bytes per cycle and SM, of the 64 there are): per 64
// columns and K block shape 1 fetches 8 KB, shape 2 16 KB, shape 3 12 KB,
// where those tiles fetch 24.  An MMA of 64 columns also takes 48 cycles for
// 32 cycles of work (it reads 6 KB of shared memory at 128 bytes per cycle);
// of 128 or more it runs at its full rate.  Leaf kernels of the 60,000 x 784
// u8 build (12 trees, 13 K blocks) 2.76 -> 1.32 ms, of 500,000 x 960 in E4M3
// (32 trees, 8 K blocks) 49.9 -> 33.3 ms.  The line between 2 and 3 (one CTA's
// four epilogue warps are too few for short rows and small leaves, where a
// larger part of the scores is kept): a K block more is worth more in shape 3 and
// what it costs besides is a leaf's, so the blocks past the fourth are weighed with
// the mean leaf.  Whole builds of 128 such leaves, 4 trees, 16 entries (32: the
// same sign or within 1.1%), shape 2 and 3 in ms:
//   8 blocks    leaves of 1,000 1.68 1.76, 1,500 2.66 2.65, 1,600 2.92 2.97,
//               1,750 3.37 3.33, 1,900 3.72 3.74
//   9 blocks    1,000 2.03 2.08, 1,250 2.58 2.57, 1,390 2.90 2.91, 1,450 3.11 3.06,
//               1,500 3.24 3.16
//   10 blocks   780 1.66 1.69, 1,000 2.15 2.14, 1,150 2.53 2.50, 1,250 2.75 2.67,
//               1,500 3.45 3.31
//   11 blocks   780 1.76 1.77, 1,000 2.28 2.25, 1,200 2.82 2.71, 1,500 3.69 3.50
//   12 blocks   780 1.85 1.81, 1,500 3.91 3.64
// and in E4M3 with 8 blocks, leaves of 1,600 3.97 3.99, 1,950 with 32 entries (500,000
// x 960, 32 trees) 62.6 60.6; with 6 blocks leaves of 1,950 3.22 3.39.
// Measured slower: A resident on one CTA per SM with 128 columns (8 blocks: 71.7
// ms per E4M3 build against 65.6 streamed), and A in Tensor Memory (such an MMA
// takes about 150 cycles at 64 columns).
bool wide_rows(int kb, int64_t leaf) { return kb >= 12 || (kb >= 8 && (kb - 4) * leaf >= 7000); }
template <int KP, int SHAPE>
struct MmaCfg {
  static constexpr int tn = SHAPE <= 1 ? 64 : (SHAPE == 2 ? 128 : 256);
  static constexpr bool stream = SHAPE >= 2;
  static constexpr int slots = KP == 16 ? 32 : 64;  // pending-key slots per row
  static constexpr int vw = SHAPE <= 2 ? 32 : 64;   // columns read from TMEM at a time
  static constexpr uint32_t stage = (stream ? kTM * 128 : 0) + tn * 128;  // bytes
  static constexpr int epi_warps = 4;
  static constexpr int threads = 32 * (epi_warps + 2);
  static constexpr int min_blocks = SHAPE == 0 ? (KP == 16 ? 3 : 2) : (SHAPE <= 2 ? 2 : 1);
};
constexpr int kMaxStages = 8;
constexpr int kColBits = 13;        // low key bits holding the column in the leaf
constexpr uint32_t kColMask = (1u << kColBits) - 1;
constexpr int kMaxLeaf = 1 << kColBits;  // largest leaf the key can address
constexpr int kCheck = 16;          // columns between flush checks

constexpr int kCentreRows = 64;     // rows averaged for a leaf's centre

__device__ __forceinline__ bool before(float da, int32_t ia, float db, int32_t ib) {
  return da < db || (da == db && (uint32_t)ia < (uint32_t)ib);
}

// ------------------------------------------------------------------ K8
template <typename T>
__device__ __forceinline__ void load4(const T *p, float *v);
template <>
__device__ __forceinline__ void load4<float>(const float *p, float *v) {
  const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <>
__device__ __forceinline__ void load4<uint8_t>(const uint8_t *p, float *v) {
  const uchar4 q = __ldg(reinterpret_cast<const uchar4 *>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}

// Streaming variants for data read or written once (evict-first in L2, so
// that the leaf centres stay resident).
template <typename T>
__device__ __forceinline__ void load4_cs(const T *p, float *v);
template <>
__device__ __forceinline__ void load4_cs<float>(const float *p, float *v) {
  const float4 q = __ldcs(reinterpret_cast<const float4 *>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <>
__device__ __forceinline__ void load4_cs<uint8_t>(const uint8_t *p, float *v) {
  const uchar4 q = __ldcs(reinterpret_cast<const uchar4 *>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}

// k_leaf_index: block (j, t) writes, for every point of leaf j of tree t,
// its position in the tree's leaf order and the leaf.
__global__ void __launch_bounds__(256) k_leaf_index(const int32_t *__restrict__ order,
                                                    const int32_t *__restrict__ goff, int64_t n,
                                                    int nleaf, int2 *__restrict__ place) {
  const int j = blockIdx.x, t = blockIdx.y;
  const int32_t *o = order + (int64_t)t * n;
  const int32_t *g = goff + (int64_t)t * (nleaf + 1);
  const int32_t lo = g[j], hi = g[j + 1];
  for (int32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const int32_t p = __ldg(o + i);
    place[(int64_t)t * n + p] = make_int2(i, j);
  }
}

// k_leaf_mean: block (j, t) for leaf j of tree t.  The centre is the mean of
// the leaf's first (up to) kCentreRows rows -- it only has to bring the
// values near zero -- summed per warp, the eight warp partials added in warp
// order, so the result does not depend on scheduling.  In both this kernel
// and k_leaf_stage lane l owns the four dimensions 4l..4l+3 of every 128-wide
// chunk (NCH chunks, d <= 128 * NCH, d % 4 == 0).
template <typename T, int NCH>
__global__ void __launch_bounds__(256) k_leaf_mean(const T *__restrict__ X, int64_t n, int d,
                                                   const int32_t *__restrict__ order,
                                                   const int32_t *__restrict__ goff, int nleaf,
                                                   float *__restrict__ mu) {
  constexpr int W = NCH * 128;
  __shared__ float part[8][W];
  const int j = blockIdx.x, t = blockIdx.y;
  const int32_t *ord = order + (int64_t)t * n;
  const int32_t *g = goff + (int64_t)t * (nleaf + 1);
  const int32_t lo = g[j], m = g[j + 1] - lo;
  if (m == 0) return;  // no point reads its centre
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float acc[NCH][4];
#pragma unroll
  for (int h = 0; h < NCH; ++h) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.0f;
  const int mc = min(m, kCentreRows);
  // warp w adds rows w, w + 8, ... in order; CB rows' loads in flight at once
  constexpr int CB = NCH <= 2 ? kCentreRows / 8 : 2;
  for (int rb = warp; rb < mc; rb += 8 * CB) {
    float v[CB][NCH][4];
#pragma unroll
    for (int i = 0; i < CB; ++i) {
      const int r = rb + 8 * i;
      const T *src = r < mc ? X + (int64_t)__ldg(ord + lo + r) * d : nullptr;
#pragma unroll
      for (int h = 0; h < NCH; ++h) {
        const int c0 = h * 128 + 4 * lane;
        v[i][h][0] = v[i][h][1] = v[i][h][2] = v[i][h][3] = 0.0f;
        if (src && c0 < d) load4<T>(src + c0, v[i][h]);
      }
    }
#pragma unroll
    for (int i = 0; i < CB; ++i)
      if (rb + 8 * i < mc)
#pragma unroll
        for (int h = 0; h < NCH; ++h)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[h][e] += v[i][h][e];
  }
#pragma unroll
  for (int h = 0; h < NCH; ++h)
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][h * 128 + 4 * lane + e] = acc[h][e];
  __syncthreads();
  float *out = mu + ((int64_t)t * nleaf + j) * d;
  for (int i = threadIdx.x; i < d; i += 256) {
    float s = 0.0f;
    for (int w = 0; w < 8; ++w) s += part[w][i];
    out[i] = s / (float)mc;
  }
}

// k_leaf_stage: warps take RB consecutive points at a time (grid-stride) and
// read their rows once; for every tree t of the chunk each point's row is
// centred on its leaf's mean and stored at its position in tree t's leaf
// order (slice t of Xq, nrm, scl).  The positions and leaves of RB points
// and up to 32 / RB trees are loaded by one lane each and broadcast.
// HBM bounds it at 128 dimensions (rows in, every tree's staged rows out; 1M x
// 128, 6 trees: 0.50 ms, 4.1 TB/s in rows of 256 bytes), issue and the latency
// of the centres' reads at wide E4M3 rows.  Visiting the points in a leaf
// order, so that a block's centres come from L1, measured slower (0.60 ms; 960
// dimensions in E4M3 11.6 against 11.0).
//
// BF16 output: the centred row rounded to BF16 (d_pad elements, zero-padded).
// E4M3 output (FP8): the centred row divided by its scale
// s = max|x - c| / 448 (448 = largest finite E4M3 value) and rounded to E4M3
// with saturation (d_pad bytes, zero-padded); the scale goes to `scl`.  In
// both cases `nrm` receives the squared norm of the row the tensor cores see
// (dequantised for FP8), so that ||y||^2 - 2 x.y ranks the same values.
// Sums of RB (a power of two, <= 32) per-lane values s[q] over the warp, all
// at once: while more than one value is left, each lane keeps half of its
// values and sends the other half to the lane that keeps those (log2 RB
// steps of RB/2, ..., 1 shuffles), then a plain butterfly over the lanes
// that hold the same value.  Lane l returns the sum for q = l >> (5 - log2 RB).
template <int RB>
__device__ __forceinline__ float warp_sum_rows(float *s, int lane) {
  int bit = 16;
#pragma unroll
  for (int cnt = RB; cnt > 1; cnt >>= 1, bit >>= 1) {
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < cnt / 2; ++i) {
      const float keep = up ? s[i + cnt / 2] : s[i];
      const float send = up ? s[i] : s[i + cnt / 2];
      s[i] = keep + __shfl_xor_sync(kFull, send, bit);
    }
  }
  float v = s[0];
#pragma unroll
  for (int o = bit; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// h * h + s for an FP16 value h, rounded once to FP32 (sm_100's multiply-add
// of FP16 factors: no conversion first).
__device__ __forceinline__ float sq_half(unsigned short h, float s) {
  float d;
  asm("fma.rn.f32.f16 %0, %1, %1, %2;" : "=f"(d) : "h"(h), "f"(s));
  return d;
}

template <int NCH>
struct StageCfg {
  static constexpr int rb = NCH <= 2 ? 4 / NCH : 1;           // points per warp step
  static constexpr int min_blocks = NCH == 1 ? 4 : (NCH == 2 ? 3 : 2);
};

// FULL: d == d_pad == 128 * NCH, so no dimension needs a bounds check.
template <typename T, int NCH, bool FP8, bool FULL>
__global__ void __launch_bounds__(256, StageCfg<NCH>::min_blocks) k_leaf_stage(const T *__restrict__ X, int64_t n, int d,
                                                    int d_pad, const int2 *__restrict__ place,
                                                    const float *__restrict__ mu, int nleaf,
                                                    int tc, void *__restrict__ Xq,
                                                    float *__restrict__ nrm,
                                                    float *__restrict__ scl) {
  constexpr int RB = StageCfg<NCH>::rb;  // points per warp step, loaded together
  constexpr int TG = 32 / RB;            // trees per broadcast group
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r0 = gw * RB; r0 < n; r0 += nw * RB) {
    float v[RB][NCH][4];
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      const int64_t r = r0 + q;
      const T *src = r < n ? X + r * d : nullptr;
#pragma unroll
      for (int h = 0; h < NCH; ++h) {
        const int c0 = h * 128 + 4 * lane;
        v[q][h][0] = v[q][h][1] = v[q][h][2] = v[q][h][3] = 0.0f;
        if (src && (FULL || c0 < d)) load4_cs<T>(src + c0, v[q][h]);
      }
    }
    for (int tg = 0; tg < tc; tg += TG) {
      int32_t my_pos = -1, my_lf = 0;
      {
        const int tt = tg + lane / RB;
        const int64_t r = r0 + lane % RB;
        if (lane < TG * RB && tt < tc && r < n) {
          const int2 pl = __ldg(place + (int64_t)tt * n + r);
          my_pos = pl.x;
          my_lf = pl.y;
        }
      }
      const int tend = min(tg + TG, tc);
      for (int t = tg; t < tend; ++t) {
        // the RB points' leaf centres are all requested before the first use
        int32_t rows[RB];
        float m4[RB][NCH][4];
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          const int src_lane = (t - tg) * RB + q;
          rows[q] = __shfl_sync(kFull, my_pos, src_lane);
          const int32_t leaf = __shfl_sync(kFull, my_lf, src_lane);  // 0 past the end
          const float *mr = mu + ((int64_t)t * nleaf + leaf) * d;
#pragma unroll
          for (int h = 0; h < NCH; ++h) {
            const int c0 = h * 128 + 4 * lane;
            m4[q][h][0] = m4[q][h][1] = m4[q][h][2] = m4[q][h][3] = 0.0f;
            if (FULL || c0 < d) load4<float>(mr + c0, m4[q][h]);
          }
        }
        float sqs[RB];  // BF16: this lane's part of each point's squared norm
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          sqs[q] = 0.0f;
          const int32_t row = rows[q];
          if (row < 0) continue;  // warp-uniform: a point past the end
          float c[NCH][4];
#pragma unroll
          for (int h = 0; h < NCH; ++h) {
            // two differences per packed FP32x2 multiply-add (-1 * m + v, one
            // rounding: the same value as v - m); past d both are 0
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const float2 r = fma2(make_float2(m4[q][h][e], m4[q][h][e + 1]),
                                    make_float2(-1.0f, -1.0f),
                                    make_float2(v[q][h][e], v[q][h][e + 1]));
              c[h][e] = r.x;
              c[h][e + 1] = r.y;
            }
          }
          const int64_t orow = (int64_t)t * n + row;
          float sq = 0.0f;
          if constexpr (FP8) {
            float amax = 0.0f;
#pragma unroll
            for (int h = 0; h < NCH; ++h)
#pragma unroll
              for (int e = 0; e < 4; ++e) amax = fmaxf(amax, fabsf(c[h][e]));
            // (not negative, so ordered as its bits)
            amax = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(amax)));
            const float sc = amax > 0.0f ? amax / 448.0f : 1.0f;
            const float inv = amax > 0.0f ? 448.0f / amax : 1.0f;
            uint8_t *dst = static_cast<uint8_t *>(Xq) + orow * d_pad;
#pragma unroll
            for (int h = 0; h < NCH; ++h) {
              const int c0 = h * 128 + 4 * lane;
              if (FULL || c0 < d_pad) {
                const __nv_fp8x2_storage_t lo2 = __nv_cvt_float2_to_fp8x2(
                    make_float2(c[h][0] * inv, c[h][1] * inv), __NV_SATFINITE, __NV_E4M3);
                const __nv_fp8x2_storage_t hi2 = __nv_cvt_float2_to_fp8x2(
                    make_float2(c[h][2] * inv, c[h][3] * inv), __NV_SATFINITE, __NV_E4M3);
                const __half2_raw a = __nv_cvt_fp8x2_to_halfraw2(lo2, __NV_E4M3);
                const __half2_raw b = __nv_cvt_fp8x2_to_halfraw2(hi2, __NV_E4M3);
                sq = sq_half(a.x, sq);
                sq = sq_half(a.y, sq);
                sq = sq_half(b.x, sq);
                sq = sq_half(b.y, sq);
                __stcs(reinterpret_cast<unsigned int *>(dst + c0),
                       (unsigned int)lo2 | ((unsigned int)hi2 << 16));
              }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(kFull, sq, o);
            if (lane == 0) {
              __stcs(nrm + orow, sq * sc * sc);
              __stcs(scl + orow, sc);
            }
          } else {
            __nv_bfloat16 *dst = static_cast<__nv_bfloat16 *>(Xq) + orow * d_pad;
            // squares of the rounded values, even and odd dimensions in the
            // two halves of a packed FP32x2 sum
            float2 sq2 = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int h = 0; h < NCH; ++h) {
              const int c0 = h * 128 + 4 * lane;
              if (FULL || c0 < d_pad) {
                const __nv_bfloat162 b01 = __floats2bfloat162_rn(c[h][0], c[h][1]);
                const __nv_bfloat162 b23 = __floats2bfloat162_rn(c[h][2], c[h][3]);
                const float2 r01 = __bfloat1622float2(b01), r23 = __bfloat1622float2(b23);
                sq2 = fma2(r01, r01, sq2);
                sq2 = fma2(r23, r23, sq2);
                uint2 pk;
                pk.x = *reinterpret_cast<const uint32_t *>(&b01);
                pk.y = *reinterpret_cast<const uint32_t *>(&b23);
                __stcs(reinterpret_cast<uint2 *>(dst + c0), pk);
              }
            }
            sqs[q] = sq2.x + sq2.y;
          }
        }
        if constexpr (!FP8) {
          // the RB norms summed over the warp together: lane l ends with
          // point (l >> (5 - log2 RB)); the first lane of each group stores it
          const float nv = warp_sum_rows<RB>(sqs, lane);
          constexpr int kGroup = 32 / RB;
          if ((lane & (kGroup - 1)) == 0) {
            const int32_t row = rows[lane / kGroup];
            if (row >= 0) __stcs(nrm + (int64_t)t * n + row, nv);
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------ K9
// Row tiles of every leaf, a block per tree, kRun consecutive leaves per
// thread and step.  One launch serves all trees (a launch per tree with one
// thread per run of leaves took 96 us each for the 32,768 leaf slots of a batch
// of 64 datasets).
__global__ void __launch_bounds__(1024) k_tile_plan(const int32_t *__restrict__ goff_all,
                                                    int nleaf, int64_t max_tiles,
                                                    int4 *__restrict__ tiles_all,
                                                    int32_t *__restrict__ n_tiles) {
  constexpr int kRun = 4;
  __shared__ int warp_tot[32];
  const int32_t *goff = goff_all + (int64_t)blockIdx.x * (nleaf + 1);
  int4 *tiles = tiles_all + (int64_t)blockIdx.x * max_tiles;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int carry = 0;
  for (int j0 = 0; j0 < nleaf; j0 += 1024 * kRun) {
    const int j1 = j0 + threadIdx.x * kRun;
    int32_t o[kRun + 1];
    int cnt = 0;
#pragma unroll
    for (int i = 0; i <= kRun; ++i) o[i] = goff[min(j1 + i, nleaf)];
#pragma unroll
    for (int i = 0; i < kRun; ++i) cnt += (o[i + 1] - o[i] + kTM - 1) / kTM;
    int x = cnt;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int y = __shfl_up_sync(kFull, x, k);
      if (lane >= k) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    int base = carry + x - cnt;
    for (int k = 0; k < 32; ++k) {
      const int y = warp_tot[k];
      if (k < w) base += y;
      carry += y;
    }
#pragma unroll
    for (int i = 0; i < kRun; ++i)
      for (int r = 0; r < o[i + 1] - o[i]; r += kTM)
        tiles[base++] = make_int4(o[i], o[i + 1] - o[i], r, j1 + i);
    __syncthreads();  // warp_tot is reused by the next step
  }
  if (threadIdx.x == 0) n_tiles[blockIdx.x] = carry;
}

// ------------------------------------------------------------------ K10
// Register-resident sorting networks (all indices compile-time constants).
__device__ __forceinline__ void cmp_swap(float *d, int32_t *id, int a, int b) {  // d[a] <= d[b]
  const bool sw = d[b] < d[a];
  const float x = d[a], y = d[b];
  const int32_t p = id[a], q = id[b];
  d[a] = sw ? y : x;
  d[b] = sw ? x : y;
  id[a] = sw ? q : p;
  id[b] = sw ? p : q;
}

// Bitonic sort, ascending.
template <int N>
__device__ __forceinline__ void bitonic_sort(float *d, int32_t *id) {
#pragma unroll
  for (int k = 2; k <= N; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int l = i ^ j;
        if (l > i) {
          if ((i & k) == 0) cmp_swap(d, id, i, l);
          else cmp_swap(d, id, l, i);
        }
      }
}

// L (ascending, N) <- the N smallest of L and S (ascending, M <= N): the
// element-wise minimum of L and reversed S is bitonic and holds them, a
// bitonic clean sorts it.
template <int N, int M>
__device__ __forceinline__ void bitonic_merge_into(float *L, int32_t *Li, const float *S,
                                                   const int32_t *Si) {
#pragma unroll
  for (int i = N - M; i < N; ++i) {
    const float sv = S[N - 1 - i];
    const int32_t si = Si[N - 1 - i];
    const bool take = sv < L[i];
    L[i] = take ? sv : L[i];
    Li[i] = take ? si : Li[i];
  }
#pragma unroll
  for (int j = N >> 1; j > 0; j >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int l = i ^ j;
      if (l > i) cmp_swap(L, Li, i, l);
    }
}

// Sorting networks on single float keys (min / max pairs).
__device__ __forceinline__ void key_cmp_swap(float *d, int a, int b) {  // d[a] <= d[b]
  const float x = fminf(d[a], d[b]), y = fmaxf(d[a], d[b]);
  d[a] = x;
  d[b] = y;
}

// Batcher's odd-even merge sort (K. E. Batcher, "Sorting networks and their
// applications", 1968), ascending: 63 exchanges for 16 keys where the bitonic
// network takes 80 (19 against 24 for 8).
template <int N>
__device__ __forceinline__ void key_sort(float *d) {
#pragma unroll
  for (int p = 1; p < N; p <<= 1)
#pragma unroll
    for (int k = p; k > 0; k >>= 1)
#pragma unroll
      for (int i = 0; i + k < N; ++i)
        if (i >= k % p && (i - k % p) % (2 * k) < k && i / (2 * p) == (i + k) / (2 * p))
          key_cmp_swap(d, i, i + k);
}

// L (ascending, N) <- the N smallest of L and S (ascending, M <= N).
template <int N, int M>
__device__ __forceinline__ void key_merge_into(float *L, const float *S) {
#pragma unroll
  for (int i = N - M; i < N; ++i) L[i] = fminf(L[i], S[N - 1 - i]);
#pragma unroll
  for (int j = N >> 1; j > 0; j >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int l = i ^ j;
      if (l > i) key_cmp_swap(L, i, l);
    }
}

// L (ascending, N) <- the N smallest of L and `key`.
template <int N>
__device__ __forceinline__ void key_insert(float *L, float key) {
  // entry i becomes max(old i - 1, min(old i, key)): every entry from the
  // old list at once, no chain through the key
  float prev = L[0];
  L[0] = fminf(prev, key);
#pragma unroll
  for (int i = 1; i < N; ++i) {
    const float cur = L[i];
    L[i] = fmaxf(prev, fminf(cur, key));
    prev = cur;
  }
}

// Shared-memory layout.  Every operand tile is rows of 128 bytes (64 BF16 or
// 128 E4M3 values of one 128-byte K block), 128-byte swizzled, 1024-byte
// aligned: resident A (kb K blocks of 16 KB), then the ring of stages.
struct MmaSmem {
  uint32_t b_off, buf_off, nrm_off, scl_off, bar_off, total;
  int stages;
};

template <int KP, int SHAPE>
__host__ __device__ inline MmaSmem mma_smem_layout(int kb, bool fp8) {
  using Cfg = MmaCfg<KP, SHAPE>;
  constexpr uint32_t rest = kTM * Cfg::slots * 4 + 2 * 4 * Cfg::tn * 4 + (2 * kMaxStages + 5) * 8 + 16;
  // a third (half, all) of the SM's 228 KB, less 1 KB per CTA for the system
  // and 1 KB to align the tiles
  constexpr uint32_t room = 228 * 1024 / Cfg::min_blocks - 2048;
  MmaSmem L;
  L.b_off = Cfg::stream ? 0 : (uint32_t)kb * kTM * 128;
  const uint32_t fixed = L.b_off + rest - (fp8 ? 0 : 4 * Cfg::tn * 4);
  const int fit = fixed < room ? (int)((room - fixed) / Cfg::stage) : 0;
  L.stages = fit < kMaxStages ? fit : kMaxStages;
  L.buf_off = L.b_off + L.stages * Cfg::stage;
  L.nrm_off = L.buf_off + kTM * (uint32_t)Cfg::slots * 4;
  L.scl_off = L.nrm_off + 4 * Cfg::tn * 4;
  L.bar_off = L.scl_off + (fp8 ? 4 * Cfg::tn * 4 : 0);
  L.total = L.bar_off + (2 * kMaxStages + 5) * 8 + 16;
  return L;
}

// KP: candidates kept per row and tree.  FP8: E4M3 operands with per-row
// scales `scl` (scores are then scaled by the row's and the column's scale);
// otherwise BF16.
template <int KP, int SHAPE, bool FP8>
__global__ void __launch_bounds__(MmaCfg<KP, SHAPE>::threads,
                                  MmaCfg<KP, SHAPE>::min_blocks) k_leaf_mma(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
    const int32_t *__restrict__ order, const float *__restrict__ nrm,
    const float *__restrict__ scl, const int4 *__restrict__ tiles,
    const int32_t *__restrict__ n_tiles, int kb, int tree, int32_t *__restrict__ run_idx,
    float *__restrict__ run_dist, int32_t *__restrict__ tree_idx, float *__restrict__ tree_dist,
    int *err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  using Cfg = MmaCfg<KP, SHAPE>;
  constexpr int kBufSlots = Cfg::slots, EPI = Cfg::epi_warps, TN = Cfg::tn;
  constexpr bool STREAM = Cfg::stream;
  const MmaSmem L = mma_smem_layout<KP, SHAPE>(kb, FP8);
  const int NS = L.stages;
  uint8_t *sA = smem;
  uint8_t *sB = smem + L.b_off;
  uint32_t *buf = reinterpret_cast<uint32_t *>(smem + L.buf_off);  // [slot][row] keys
  float *nbuf = reinterpret_cast<float *>(smem + L.nrm_off);  // [warp][TN] column norms of a tile
  float *sbuf = reinterpret_cast<float *>(smem + L.scl_off);  // [warp][TN] column scales (FP8)
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bar_off);
  uint64_t *full_a = bars + 0;
  uint64_t *acc_full = bars + 1;   // 2 accumulators
  uint64_t *acc_empty = bars + 3;  // 2 accumulators
  uint64_t *full_b = bars + 5;     // NS stages
  uint64_t *empty_b = full_b + kMaxStages;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(empty_b + kMaxStages);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  constexpr int kKE = FP8 ? 128 : 64;  // elements per 128-byte K block
  constexpr uint32_t kStageA = STREAM ? kTM * 128 : 0;

  const int u = blockIdx.x;
  if (u >= *n_tiles) return;  // uniform for the whole block
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int4 tile = __ldg(tiles + u);
  const int32_t lo = tile.x, m = tile.y;
  const int r0 = tile.z;
  if (m > kMaxLeaf) {  // the candidate keys address at most kMaxLeaf columns
    if (threadIdx.x == 0) atomicOr(err, 2);
    empty_lists<KP>(order + lo + r0, min(kTM, m - r0), tree > 0 ? tree_idx : run_idx,
                    tree > 0 ? tree_dist : run_dist);
    return;  // uniform for the whole block
  }
  const int nct = (m + TN - 1) / TN;

  if (threadIdx.x == 0) {
    mbar_init(full_a, 1);
    for (int s = 0; s < NS; ++s) {
      mbar_init(full_b + s, 1);
      mbar_init(empty_b + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + b, 1);
      mbar_init(acc_empty + b, EPI * 32);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == EPI + 1) tmem_alloc(tmem_slot, 2 * TN);
  if (warp == EPI && lane == 0) {
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == EPI) {
    // ---- TMA producer: stage i = (column tile c, K block q), i = c * kb + q
    if (elect_one()) {
      if constexpr (!STREAM) {
        mbar_arrive_expect_tx(full_a, (uint32_t)kb * kTM * 128);
        for (int q = 0; q < kb; ++q)
          tma_load_2d(sA + q * kTM * 128, &tmA, full_a, q * kKE, lo + r0);
      }
      const int total = nct * kb;
      int s = 0, ph = 1, q = 0, y = lo;
      for (int i = 0; i < total && !*abort_flag; ++i) {
        if (i >= NS && !mbar_wait(empty_b + s, ph)) {
          *abort_flag = 1;
          break;
        }
        uint8_t *st = sB + s * Cfg::stage;
        mbar_arrive_expect_tx(full_b + s, Cfg::stage);
        if constexpr (STREAM) tma_load_2d(st, &tmA, full_b + s, q * kKE, lo + r0);
        tma_load_2d(st + kStageA, &tmB, full_b + s, q * kKE, y);
        if (++s == NS) {
          s = 0;
          ph ^= 1;
        }
        if (++q == kb) {
          q = 0;
          y += TN;
        }
      }
    }
  } else if (warp == EPI + 1) {
    // ---- MMA issuer: 4 instructions per 128-byte K block (K = 16 BF16 or
    // 32 E4M3 values, 32 bytes each).  It shares its issue slots with epilogue
    // warps: as the elected lane instead of lane 0 (descriptors in uniform
    // registers) it brought the leaves of 250,000 x 256, 16 trees from 3.47 to
    // 3.02 ms, 60,000 x 784 1%; 1M x 128, two K blocks, takes 0.5% longer.
    if (elect_one()) {
      constexpr uint32_t idesc = FP8 ? idesc_e4m3_f32(kTM, TN) : idesc_bf16_f32(kTM, TN);
      const uint32_t a_base = smem_u32(sA), b_base = smem_u32(sB);
      bool ok = STREAM || mbar_wait(full_a, 0);
      int s = 0, ph = 0;
      for (int c = 0; ok && c < nct && !*abort_flag; ++c) {
        const int b = c & 1;
        if (c > 1) ok = mbar_wait(acc_empty + b, ((c >> 1) - 1) & 1);
        for (int q = 0; ok && q < kb; ++q) {
          ok = mbar_wait(full_b + s, ph);
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = b_base + s * Cfg::stage;
          const uint64_t ad = desc_k_sw128(STREAM ? st : a_base + q * kTM * 128);
          const uint64_t bd = desc_k_sw128(st + kStageA);
#pragma unroll
          for (int k = 0; k < 4; ++k) {  // 32 bytes further: 2 in the descriptors' address
            if constexpr (FP8)
              mma_e4m3(tmem + b * TN, ad + 2 * k, bd + 2 * k, idesc, (q | k) ? 1u : 0u);
            else
              mma_bf16(tmem + b * TN, ad + 2 * k, bd + 2 * k, idesc, (q | k) ? 1u : 0u);
          }
          mma_commit(empty_b + s);
          if (++s == NS) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok) mma_commit(acc_full + b);
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    // ---- epilogue: thread = row (TMEM lane).  A candidate is one 32-bit
    // key: its score (an FP32 value, ordered as a float) with the low
    // kColBits mantissa bits replaced by its column in the leaf, so keys sort
    // with plain min/max and equal scores order by column.  Keys below the
    // row's current KP-th best go to a slot-major shared buffer
    // (conflict-free: consecutive rows are consecutive words); when any row
    // of the warp has too many pending, every row sorts its pending keys in
    // batches and merges them into its sorted list of KP keys.
    const int row = warp * 32 + lane;
    const bool rvalid = r0 + row < m;
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    float td[KP];
#pragma unroll
    for (int j = 0; j < KP; ++j) td[j] = __int_as_float(0x7f800000);
    // Candidates that cannot beat the KP-th of the point's running list
    // (approximate squared distances of the earlier trees) are never kept.
    // (rows past the leaf get -inf and keep nothing)
    float thr = rvalid ? __int_as_float(0x7f800000) : -__int_as_float(0x7f800000);
    int32_t my_pos = -1, my_pt = -1;
    float nr = 0.0f, m2s = -2.0f;  // FP8: -2 x the row's scale
    if (rvalid) {
      my_pos = lo + r0 + row;
      my_pt = __ldg(order + my_pos);
      nr = __ldg(nrm + my_pos);
      if constexpr (FP8) m2s = -2.0f * __ldg(scl + my_pos);
      if (tree > 0) thr = run_dist[(int64_t)my_pt * KP + KP - 1] - nr;
    }
    const float thr0 = thr;
    // Pending keys: a passing key is stored at the next free slot of one of
    // two per-row lanes of the buffer (even and odd columns, two independent
    // append chains) by a predicated shared-memory store, no branch; slot
    // addresses are 32-bit shared-window offsets.
    constexpr int kChains = 2, kLane = kBufSlots / kChains, kPerBatch = 16 / kChains;
    uint32_t *const pbase = buf + row;
    const uint32_t abase = smem_u32(pbase);
    uint32_t aslot[kChains], alim[kChains];
#pragma unroll
    for (int q = 0; q < kChains; ++q) {
      aslot[q] = abase + q * kLane * kTM * 4;
      // after a check that does not flush a chain holds at most
      // kLane - kCheck / kChains keys, so the next kCheck / kChains stores
      // stay inside its kLane slots
      alim[q] = aslot[q] + (kLane - kCheck / kChains) * kTM * 4;
    }
    // The flush is a few hundred instructions of unrolled networks.  The scan
    // below is written so that the kernel holds one copy of it: with a copy at
    // every check (nine) the warps waited for instructions.  With the shorter
    // networks, the one-instruction key and the predicated append: 121.5 M ->
    // 99 M warp instructions per tree at 262,144 x 128, 213 -> 185 us under
    // the profiler; the 1M x 128 build of 6 trees 7.20 -> 6.76 ms.
    const int own = r0 + warp * 32;  // columns own .. own + 31: the warp's own points
    int seen = 0;                    // columns below it are flushed
    auto flush = [&](int upto) {
      int cnt[kChains], mx = 0;
#pragma unroll
      for (int q = 0; q < kChains; ++q) {
        cnt[q] = (int)((aslot[q] - abase) / (kTM * 4)) - q * kLane;
        mx = max(mx, cnt[q]);
      }
      mx = __reduce_max_sync(kFull, mx);
      if (own < upto && own + 32 > seen) {
        // the row's own point may be pending (in one of the row's tiles):
        // its key becomes infinite (eight slots read at a time; those past
        // the pending ones are not changed)
#pragma unroll 1
        for (int e0 = 0; e0 < mx; e0 += 4) {
          uint32_t key[4][kChains];
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int q = 0; q < kChains; ++q) key[e][q] = pbase[(q * kLane + e0 + e) * kTM];
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int q = 0; q < kChains; ++q)
              if (e0 + e < cnt[q] && (key[e][q] & kColMask) == (uint32_t)(own + lane))
                pbase[(q * kLane + e0 + e) * kTM] = 0x7f800000u;
        }
      }
      seen = upto;
      // W keys of each chain from slot `base` on (+inf past its pending
      // ones), sorted and merged into the list
      auto take = [&](int base, auto width) {
        constexpr int W = decltype(width)::value;
        float sd[kChains * W];
#pragma unroll
        for (int q = 0; q < kChains; ++q)
#pragma unroll
          for (int e = 0; e < W; ++e) {
            sd[q * W + e] = __int_as_float(0x7f800000);
            if (base + e < cnt[q])
              sd[q * W + e] = __uint_as_float(pbase[(q * kLane + base + e) * kTM]);
          }
        key_sort<kChains * W>(sd);
        key_merge_into<KP, kChains * W>(td, sd);
      };
      int base = 0;
      constexpr int kTail = KP == 16 ? 3 : 2;
#pragma unroll 1
      for (; mx - base > kTail; base += kPerBatch)
        take(base, std::integral_constant<int, kPerBatch>{});
      // a rest of a few keys a chain one by one (2 KP min/max each): cheaper
      // than a batch of 16 and its merge (about 200); the kept keys are the same
#pragma unroll 1
      for (; base < mx; ++base)
#pragma unroll
        for (int q = 0; q < kChains; ++q) {
          float key = __int_as_float(0x7f800000);
          if (base < cnt[q]) key = __uint_as_float(pbase[(q * kLane + base) * kTM]);
          key_insert<KP>(td, key);
        }
#pragma unroll
      for (int q = 0; q < kChains; ++q) aslot[q] = abase + q * kLane * kTM * 4;
      thr = fminf(thr0, td[KP - 1]);
    };
    // key = the score's high bits and the column bits of the packed norm
    // (one bit-select), stored only when the score beats the threshold
    auto append = [&](uint32_t &slot, float sv, float ncp) {
      uint32_t key;  // one bit-select (0xD8: sv where the mask is 0, else ncp)
      asm("lop3.b32 %0, %1, %2, %3, 0xD8;"
          : "=r"(key)
          : "r"(__float_as_uint(sv)), "r"(__float_as_uint(ncp)), "r"(kColMask));
      if (sv < thr) {  // becomes two predicated instructions
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(slot), "r"(key) : "memory");
        slot += kTM * 4;
      }
    };
    // kCheck columns of scores; their packed norms (and E4M3 scales) are read
    // into registers before the stores, so the loads do not wait behind them.
    // Returns whether a chain is too full for another kCheck columns.
    auto scan = [&](const float *v, const float *wn, const float *ws) {
      float nc[kCheck], sc[kCheck];
#pragma unroll
      for (int j4 = 0; j4 < kCheck; j4 += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(wn + j4);
        nc[j4] = a.x;
        nc[j4 + 1] = a.y;
        nc[j4 + 2] = a.z;
        nc[j4 + 3] = a.w;
        if constexpr (FP8) {
          const float4 b = *reinterpret_cast<const float4 *>(ws + j4);
          sc[j4] = b.x;
          sc[j4 + 1] = b.y;
          sc[j4 + 2] = b.z;
          sc[j4 + 3] = b.w;
        }
      }
      (void)sc;
#pragma unroll
      for (int e = 0; e < kCheck; e += 2) {
        float2 sv;
        if constexpr (FP8) {
          sv.x = fmaf(m2s * sc[e], v[e], nc[e]);
          sv.y = fmaf(m2s * sc[e + 1], v[e + 1], nc[e + 1]);
        } else {
          // two scores per packed FP32x2 multiply-add
          sv = fma2(make_float2(v[e], v[e + 1]), make_float2(-2.0f, -2.0f),
                    make_float2(nc[e], nc[e + 1]));
        }
        append(aslot[e % kChains], sv.x, nc[e]);
        append(aslot[(e + 1) % kChains], sv.y, nc[e + 1]);
      }
      bool over = false;
#pragma unroll
      for (int q = 0; q < kChains; ++q) over |= aslot[q] > alim[q];
      return over;
    };
    // column norms (and E4M3 scales) of a tile: lane l holds columns l and
    // l + 32, loaded one tile ahead; columns past the leaf carry an infinite
    // norm (a NaN once packed) and so never pass
    float pn[TN / 32], ps[TN / 32];
    auto load_cols = [&](int c) {
#pragma unroll
      for (int h = 0; h < TN / 32; ++h) {
        const int col = c * TN + h * 32 + lane;
        const bool in = c < nct && col < m;
        pn[h] = in ? __ldg(nrm + lo + col) : __int_as_float(0x7f800000);
        ps[h] = 0.0f;
        if constexpr (FP8) ps[h] = in ? __ldg(scl + lo + col) : 0.0f;
      }
    };
    load_cols(0);
    float *wn = nbuf + warp * TN;
    float *ws = sbuf + warp * TN;
#pragma unroll 1
    for (int c = 0; c < nct; ++c) {
      const int b = c & 1;
      // this tile's column norms, staged per warp (16-byte aligned reads)
      __syncwarp();
#pragma unroll
      for (int h = 0; h < TN / 32; ++h) {
        // the norm's low kColBits bits replaced by the column (a relative
        // change below 2^-10 of the norm, next to the BF16 rounding of x.y);
        // a past-the-leaf column's infinite norm becomes a NaN, which
        // fails every comparison
        wn[h * 32 + lane] = __uint_as_float((__float_as_uint(pn[h]) & ~kColMask) |
                                            (uint32_t)(c * TN + h * 32 + lane));
        if constexpr (FP8) ws[h * 32 + lane] = ps[h];
      }
      __syncwarp();
      load_cols(c + 1);
      if (!__all_sync(kFull, mbar_wait(acc_full + b, (c >> 1) & 1))) {
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      constexpr int VW = Cfg::vw;
#pragma unroll 1
      for (int q = 0; q < TN; q += VW) {
        float v[VW];
#pragma unroll
        for (int i = 0; i < VW; i += 32) tmem_ld32(lane_base + b * TN + q + i, v + i);
        if (q + VW == TN) {  // the accumulator is in registers: the next tile may have it
          tc_fence_before();
          mbar_arrive(acc_empty + b);
        }
        // groups of kCheck columns, one after the other; a group that leaves a
        // chain too full goes to the one flush and on with the next group
        auto group = [&](int g) {
          return __any_sync(kFull, scan(v + g * kCheck, wn + q + g * kCheck,
                                        ws + q + g * kCheck)) != 0;
        };
        const int done = c * TN + q;
        if constexpr (VW == 32) {
          bool last = false;
          if (!group(0)) goto second;
        full:
          flush(done + (last ? 32 : kCheck));
          if (last) continue;
        second:
          last = true;
          if (group(1) || done + 32 == nct * TN) goto full;
        } else {
          int h = 0;
        next:
          bool over = false;
          switch (h) {
            case 0:
              h = kCheck;
              if ((over = group(0))) break;
              [[fallthrough]];
            case kCheck:
              h = 2 * kCheck;
              if ((over = group(1))) break;
              [[fallthrough]];
            case 2 * kCheck:
              h = 3 * kCheck;
              if ((over = group(2))) break;
              [[fallthrough]];
            default:
              h = 4 * kCheck;
              over = group(3);
          }
          if (over || done + h == nct * TN) flush(done + h);
          if (h < VW) goto next;
        }
      }
    }
    if (rvalid) {
      // this tree's list, keys back to (squared distance, point id), already
      // ascending by key, i.e. by distance: tree 0's is the running list;
      // later trees' go to the tree list, which k_fold_lists merges into the
      // running list (a separate, fully parallel pass: folding here kept the
      // CTA, its idle TMA and MMA warps and its shared memory for the
      // latency of the running list's reads)
      float rd[KP];
      int32_t ri[KP];
#pragma unroll
      for (int j = 0; j < KP; ++j) {
        const uint32_t key = __float_as_uint(td[j]);
        // (a score of -inf, its column's bits set, is a NaN, of which the networks
        // make one with all bits set: no column of the leaf)
        const bool have = key != 0x7f800000u && (int)(key & kColMask) < m;
        const int32_t q = have ? __ldg(order + lo + (int32_t)(key & kColMask)) : -1;
        rd[j] = have ? nr + __uint_as_float(key & ~kColMask) : __int_as_float(0x7f800000);
        ri[j] = q;
      }
      const int64_t o = (int64_t)my_pt * KP;
      float4 *dd = reinterpret_cast<float4 *>((tree > 0 ? tree_dist : run_dist) + o);
      int4 *di = reinterpret_cast<int4 *>((tree > 0 ? tree_idx : run_idx) + o);
#pragma unroll
      for (int j = 0; j < KP; j += 4) {
        dd[j / 4] = make_float4(rd[j], rd[j + 1], rd[j + 2], rd[j + 3]);
        di[j / 4] = make_int4(ri[j], ri[j + 1], ri[j + 2], ri[j + 3]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == EPI + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 2 * TN);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicOr(err, 1);
}

// k_fold_lists: per point (one thread each), fold this tree's list (KP
// candidates ascending by approximate distance) into the running list of the
// KP best distinct candidates of the trees before: neighbours the running
// list already holds are dropped from the new list, which is re-sorted, and a
// bitonic merge keeps the KP best by distance.
//
// A warp's 32 lists of one array are consecutive: it loads and stores them 512
// bytes at a time and turns them (a lane's list <-> 32 consecutive 16-byte pieces)
// through 4 KB of shared memory of its own, 16-byte piece c of point p at c ^ p
// (c ^ p / 2 with four pieces a point), which uses all banks both ways.  A lane
// reading its own 128-byte list took 32 cache lines per load: 64 uneven sets of
// 96 dimensions, 32 entries 545 -> 504 us a tree, 500,000 points 119 -> 113, 1M
// points with 16 entries 73 -> 68.  With 32 entries the duplicate search and the
// networks, 2,900 half-rate instructions a point, bound it; with 16, HBM.
constexpr int kFoldThreads = 128;
template <int KP>
__global__ void __launch_bounds__(kFoldThreads) k_fold_lists(const float *__restrict__ tree_dist,
                                                             const int32_t *__restrict__ tree_idx,
                                                             int64_t n,
                                                             float *__restrict__ run_dist,
                                                             int32_t *__restrict__ run_idx) {
  constexpr int Q = KP / 4;  // 16-byte pieces of a list
  __shared__ uint4 turn[kFoldThreads / 32][32 * Q];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t p0 = (int64_t)blockIdx.x * kFoldThreads + 32 * warp;
  if (p0 >= n) return;  // the whole warp
  const int pieces = (int)min64(32, n - p0) * Q;
  uint4 *buf = turn[warp];
  const auto slot = [](int p, int c) { return p * Q + (c ^ (Q == 8 ? p & 7 : (p >> 1) & 3)); };
  const auto fetch = [&](const void *list, bool last_use, uint4 *v) {
    const uint4 *src = static_cast<const uint4 *>(list) + p0 * Q;
#pragma unroll
    for (int i = 0; i < Q; ++i)
      if (32 * i + lane < pieces) {
        if (last_use) v[i] = __ldcs(src + 32 * i + lane);
        else v[i] = src[32 * i + lane];
      }
  };
  const auto to_lists = [&](uint4 *v) {
#pragma unroll
    for (int i = 0; i < Q; ++i) buf[slot((32 * i + lane) / Q, lane % Q)] = v[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < Q; ++i) v[i] = buf[slot(lane, i)];
    __syncwarp();
  };
  const auto put = [&](const uint4 *v, void *list) {
    uint4 *dst = static_cast<uint4 *>(list) + p0 * Q;
#pragma unroll
    for (int i = 0; i < Q; ++i) buf[slot(lane, i)] = v[i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < Q; ++i)
      if (32 * i + lane < pieces) dst[32 * i + lane] = buf[slot((32 * i + lane) / Q, lane % Q)];
    __syncwarp();
  };
  uint4 w[4][Q];  // lanes past the last point fold what lies there and write nothing
  fetch(tree_dist, true, w[0]);
  fetch(tree_idx, true, w[1]);
  fetch(run_dist, false, w[2]);
  fetch(run_idx, false, w[3]);
#pragma unroll
  for (int a = 0; a < 4; ++a) to_lists(w[a]);
  float rd[KP], od[KP];
  int32_t ri[KP], oi[KP];
#pragma unroll
  for (int j = 0; j < KP; j += 4) {
    const uint4 a = w[0][j / 4], b = w[1][j / 4], c = w[2][j / 4], e = w[3][j / 4];
    rd[j] = __uint_as_float(a.x); rd[j + 1] = __uint_as_float(a.y);
    rd[j + 2] = __uint_as_float(a.z); rd[j + 3] = __uint_as_float(a.w);
    ri[j] = b.x; ri[j + 1] = b.y; ri[j + 2] = b.z; ri[j + 3] = b.w;
    od[j] = __uint_as_float(c.x); od[j + 1] = __uint_as_float(c.y);
    od[j + 2] = __uint_as_float(c.z); od[j + 3] = __uint_as_float(c.w);
    oi[j] = e.x; oi[j + 1] = e.y; oi[j + 2] = e.z; oi[j + 3] = e.w;
  }
#pragma unroll
  for (int j = 0; j < KP; ++j) {
    bool dup = false;
#pragma unroll
    for (int i = 0; i < KP; ++i) dup |= (ri[j] >= 0 && oi[i] == ri[j]);
    if (dup) {
      ri[j] = -1;
      rd[j] = __int_as_float(0x7f800000);
    }
  }
  bitonic_sort<KP>(rd, ri);
  bitonic_merge_into<KP, KP>(od, oi, rd, ri);
#pragma unroll
  for (int j = 0; j < KP; j += 4) {
    w[0][j / 4] = make_uint4(__float_as_uint(od[j]), __float_as_uint(od[j + 1]),
                             __float_as_uint(od[j + 2]), __float_as_uint(od[j + 3]));
    w[1][j / 4] = make_uint4(oi[j], oi[j + 1], oi[j + 2], oi[j + 3]);
  }
  put(w[0], run_dist);
  put(w[1], run_idx);
}

// The same with KP lanes per point, the lists' entries one per lane: the same
// networks exchange over shuffles, so the lists (equal distances included) come
// out the same.  For few points, where a thread per point leaves most of the
// GPU idle and its ~2,000 dependent operations set the time (2,003 points, 32
// entries: 10.5 us, these lanes 3.1); it issues twice the instructions (31,337
// points, 16 entries: 7.3 us against 5.2), hence kFoldLanes.
template <int KP>
__global__ void __launch_bounds__(256) k_fold_lanes(const float *__restrict__ tree_dist,
                                                    const int32_t *__restrict__ tree_idx,
                                                    int64_t n, float *__restrict__ run_dist,
                                                    int32_t *__restrict__ run_idx) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = e < n * KP;  // KP lanes of a point alike
  const int p = threadIdx.x & (KP - 1);
  const float inf = __int_as_float(0x7f800000);
  float rd = live ? __ldcs(tree_dist + e) : inf, od = live ? run_dist[e] : inf;
  int32_t ri = live ? __ldcs(tree_idx + e) : -1, oi = live ? run_idx[e] : -1;
  bool dup = false;
#pragma unroll
  for (int i = 0; i < KP; ++i) dup |= __shfl_sync(kFull, oi, i, KP) == ri;
  if (dup && ri >= 0) {
    ri = -1;
    rd = inf;
  }
  // entry p and its partner p ^ j, ascending (up) or descending
  auto exchange = [&](float &d, int32_t &id, int j, bool up) {
    const float q = __shfl_xor_sync(kFull, d, j, KP);
    const int32_t qi = __shfl_xor_sync(kFull, id, j, KP);
    const bool low = (p & j) == 0;
    if (low == up ? q < d : d < q) {
      d = q;
      id = qi;
    }
  };
#pragma unroll
  for (int k = 2; k <= KP; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) exchange(rd, ri, j, (p & k) == 0);
  const float sv = __shfl_sync(kFull, rd, KP - 1 - p, KP);
  const int32_t si = __shfl_sync(kFull, ri, KP - 1 - p, KP);
  if (sv < od) {
    od = sv;
    oi = si;
  }
#pragma unroll
  for (int j = KP >> 1; j > 0; j >>= 1) exchange(od, oi, j, true);
  if (live) {
    run_dist[e] = od;
    run_idx[e] = oi;
  }
}

// ------------------------------------------------------------------ K11
// One warp per point.  d <= 256: four candidates at a time, eight lanes
// each, every lane reading 16-byte pieces of the candidate row (a group reads
// 128 contiguous bytes per load); d > 256: one candidate at a time over the
// whole warp (lane l holds dimensions 4l..4l+3 of every 128-wide chunk).
// Each lane adds its squared differences with fused multiply-adds and a
// fixed butterfly adds the lane sums: an FP32 distance with pairwise
// summation, the same on every run.  Lane j then holds candidate j (j < K2)
// and the K2 pairs are sorted with a bitonic network; candidates whose
// distance lies within 2^-16 of the k-th are re-ordered by an FP64
// distance.  d must be a multiple of 4.
template <typename T, int D, int K2>
__global__ void __launch_bounds__(256) k_rerank(const T *__restrict__ X, int d,
                                                const int32_t *__restrict__ visit, int64_t n,
                                                const int32_t *__restrict__ ci, int k,
                                                int32_t *__restrict__ oi, float *__restrict__ od) {
  const int lane = threadIdx.x & 31;
  const int g = 0, j = lane;  // one point per warp: the group is the warp
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n) return;  // warp-uniform
  const bool live = true;
  const int32_t p = visit ? __ldg(visit + w) : (int32_t)w;
  const float inf = __int_as_float(0x7f800000);
  const int32_t c = lane < K2 ? __ldg(ci + (int64_t)p * K2 + lane) : -1;
  float dist = inf;
  if constexpr (D <= 256) {
    // four candidates per pass, eight lanes each: lane s of group g holds
    // dimensions 4s + 32t .. +3 (t < D / 32) of the query and adds the
    // squared differences of those dimensions of candidate 4 pass + g; a
    // fixed butterfly over the group's lanes completes the sum
    constexpr int NQ = D / 32;
    const int grp = lane >> 3, sl = lane & 7;
    float q[NQ][4];
    const T *xp = X + (int64_t)p * d;
#pragma unroll
    for (int t = 0; t < NQ; ++t) {
      const int c0 = 32 * t + 4 * sl;
      q[t][0] = q[t][1] = q[t][2] = q[t][3] = 0.0f;
      if (c0 < d) load4<T>(xp + c0, q[t]);
    }
#pragma unroll
    for (int pass = 0; pass < K2 / 4; ++pass) {
      const int32_t cj = __shfl_sync(kFull, c, 4 * pass + grp);
      float acc = 0.0f;
      if (cj >= 0) {
        const T *xc = X + (int64_t)cj * d;
#pragma unroll
        for (int t = 0; t < NQ; ++t) {
          const int c0 = 32 * t + 4 * sl;
          if (c0 < d) {
            float v[4];
            load4<T>(xc + c0, v);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float df = v[e] - q[t][e];
              acc = fmaf(df, df, acc);
            }
          }
        }
      }
      acc += __shfl_xor_sync(kFull, acc, 4);
      acc += __shfl_xor_sync(kFull, acc, 2);
      acc += __shfl_xor_sync(kFull, acc, 1);
      const float got = __shfl_sync(kFull, acc, 8 * (lane & 3));
      if ((lane >> 2) == pass && c >= 0) dist = sqrtf(got);
    }
  } else {
    constexpr int NC = (D + 127) / 128;  // 128-wide chunks (d <= D <= 1024)
    float q[NC][4];
    const T *xp = X + (int64_t)p * d;
#pragma unroll
    for (int h = 0; h < NC; ++h) {
      const int c0 = h * 128 + 4 * lane;
      q[h][0] = q[h][1] = q[h][2] = q[h][3] = 0.0f;
      if (c0 < d) load4<T>(xp + c0, q[h]);
    }
#pragma unroll 4
    for (int jj = 0; jj < K2; ++jj) {
      const int32_t cj = __shfl_sync(kFull, c, jj);
      if (cj < 0) continue;  // warp-uniform
      const T *xc = X + (int64_t)cj * d;
      float acc = 0.0f;
#pragma unroll
      for (int h = 0; h < NC; ++h) {
        const int c0 = h * 128 + 4 * lane;
        if (c0 < d) {
          float v[4];
          load4<T>(xc + c0, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float df = v[e] - q[h][e];
            acc = fmaf(df, df, acc);
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
      if (lane == jj) dist = sqrtf(acc);
    }
  }
  int32_t id = c;
  // bitonic sort of K2 (dist, id) pairs inside the group, ascending
#pragma unroll
  for (int size = 2; size <= K2; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const float od_ = __shfl_xor_sync(kFull, dist, stride);
      const int32_t oi_ = __shfl_xor_sync(kFull, id, stride);
      const bool up = ((j & size) == 0);
      const bool lower = (j & stride) == 0;
      const bool mine_first = before(dist, id, od_, oi_);
      const bool keep = (lower == up) ? mine_first : !mine_first;
      if (!keep) {
        dist = od_;
        id = oi_;
      }
    }
  }
  // FP64 check of the candidates near the k-th distance
  const float dk = __shfl_sync(kFull, dist, g * K2 + k - 1);
  const float eps = 1.52587890625e-05f;  // 2^-16
  const bool near = id >= 0 && isfinite(dk) && fabsf(dist - dk) <= eps * dk;
  const unsigned gmask = (K2 == 32 ? 0xffffffffu : ((1u << K2) - 1u)) << (g * K2);
  const unsigned wmask = __ballot_sync(kFull, near) & gmask;
  const unsigned below = gmask & ((1u << (g * K2 + k)) - 1u);
  if (__any_sync(kFull, (wmask & below) != 0 && (wmask & ~below) != 0)) {
    const bool act = (wmask & below) != 0 && (wmask & ~below) != 0;  // group-uniform
    double d64 = 1e300;
    if (act && near) {
      const T *xp = X + (int64_t)p * d, *xc = X + (int64_t)id * d;
      double s = 0.0;
      for (int i = 0; i < d; ++i) {
        const double df = (double)xc[i] - (double)xp[i];
        s += df * df;
      }
      d64 = sqrt(s);
    }
    // re-order the window by (FP64 distance, id); other lanes keep their place
    const int first = act ? __ffs(wmask) - 1 : lane;
    int rank = 0;
    for (int q = 0; q < 32; ++q) {
      const double oq = __shfl_sync(kFull, d64, q);
      const int32_t iq = __shfl_sync(kFull, id, q);
      if (act && near && ((wmask >> q) & 1u) &&
          (oq < d64 || (oq == d64 && (uint32_t)iq < (uint32_t)id)))
        ++rank;
    }
    const int dest = (act && near) ? first + rank : lane;
    float nd = dist;
    int32_t ni = id;
    for (int q = 0; q < 32; ++q) {
      const int dq = __shfl_sync(kFull, dest, q);
      const float dv = __shfl_sync(kFull, dist, q);
      const int32_t iv = __shfl_sync(kFull, id, q);
      if (act && ((wmask >> q) & 1u) && dq == lane) {
        nd = dv;
        ni = iv;
      }
    }
    dist = nd;
    id = ni;
  }
  if (live && j < k) {
    oi[(int64_t)p * k + j] = id;
    od[(int64_t)p * k + j] = id >= 0 ? dist : inf;
  }
}

template <typename T, int D, int K2>
drpt_status launch_rerank_t(const void *X, int d, const int32_t *visit, int64_t n,
                            const int32_t *cand, int k, int32_t *out_idx, float *out_dist,
                            cudaStream_t s) {
  const int64_t warps = n;
  const unsigned grid = (unsigned)ceil_div(warps * 32, 256);
  k_rerank<T, D, K2><<<grid, 256, 0, s>>>((const T *)X, d, visit, n, cand, k, out_idx, out_dist);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

template <typename T, int K2>
drpt_status launch_rerank_d(const void *X, int d, const int32_t *visit, int64_t n,
                            const int32_t *cand, int k, int32_t *out_idx, float *out_dist,
                            cudaStream_t s) {
  // D: an upper bound of d in whole 128-value chunks (the kernel guards c0 < d)
  if (d <= 128) return launch_rerank_t<T, 128, K2>(X, d, visit, n, cand, k, out_idx, out_dist, s);
  if (d <= 256) return launch_rerank_t<T, 256, K2>(X, d, visit, n, cand, k, out_idx, out_dist, s);
  if (d <= 512) return launch_rerank_t<T, 512, K2>(X, d, visit, n, cand, k, out_idx, out_dist, s);
  return launch_rerank_t<T, 1024, K2>(X, d, visit, n, cand, k, out_idx, out_dist, s);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

drpt_status make_tmap(CUtensorMap *map, const void *base, int64_t rows, int d_pad, int box_rows,
                      bool fp8) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available");
    return DRPT_ERR_CUDA;
  }
  const int esz = fp8 ? 1 : 2;
  cuuint64_t dims[2] = {(cuuint64_t)d_pad, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)d_pad * esz};
  cuuint32_t box[2] = {(cuuint32_t)(128 / esz), (cuuint32_t)box_rows};  // 128-byte rows
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  const_cast<void *>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
    return DRPT_ERR_CUDA;
  }
  return DRPT_OK;
}

template <typename T, int NCH>
void stage_t(const LeafStageArgs &a, bool means, cudaStream_t s) {
  const T *X = (const T *)a.X;
  if (means) {
    const dim3 g((unsigned)a.nleaf, (unsigned)a.T);
    k_leaf_index<<<g, 256, 0, s>>>(a.order, a.goff, a.n, a.nleaf, a.place);
    k_leaf_mean<T, NCH><<<g, 256, 0, s>>>(X, a.n, a.d, a.order, a.goff, a.nleaf, a.mu);
    return;
  }
  constexpr int RB = StageCfg<NCH>::rb;
  // one resident round of blocks, each warp looping over its points
  const bool full = a.d == NCH * 128 && a.d_pad == NCH * 128;
  auto kern = a.fp8 ? (full ? k_leaf_stage<T, NCH, true, true> : k_leaf_stage<T, NCH, true, false>)
                    : (full ? k_leaf_stage<T, NCH, false, true> : k_leaf_stage<T, NCH, false, false>);
  static int per_sm = 0;  // the four forms use the same registers within a few
  if (per_sm == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0) != cudaSuccess ||
        per_sm < 1)
      per_sm = 1;
  }
  const int sms = device_sm_count();
  const unsigned grid =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(a.n, 8 * RB), (int64_t)sms * per_sm));
  const int64_t toff = (int64_t)a.t0 * a.n;
  const float *mu = a.mu + (int64_t)a.t0 * a.nleaf * a.d;
  kern<<<grid, 256, 0, s>>>(X, a.n, a.d, a.d_pad, a.place + toff, mu, a.nleaf, a.tc, a.Xb, a.nrm,
                            a.scl);
}

template <typename T>
void stage_d(const LeafStageArgs &a, bool means, cudaStream_t s) {
  if (a.d_pad <= 128) stage_t<T, 1>(a, means, s);
  else if (a.d_pad <= 256) stage_t<T, 2>(a, means, s);
  else if (a.d_pad <= 512) stage_t<T, 4>(a, means, s);
  else stage_t<T, 8>(a, means, s);
}

template <int KP, int SHAPE, bool FP8>
drpt_status mma_t(const MixedTreeArgs &a, const CUtensorMap &tmA, int kb, cudaStream_t s) {
  using Cfg = MmaCfg<KP, SHAPE>;
  CUtensorMap tmB;
  DRPT_TRY(make_tmap(&tmB, a.Xb, a.n, a.d_pad, Cfg::tn, a.fp8));
  const MmaSmem L = mma_smem_layout<KP, SHAPE>(kb, FP8);
  const size_t smem = L.total + 1024;
  if (L.stages < 1) {
    set_error("mixed leaf kernel: no room for %d K blocks", kb);
    return DRPT_ERR_UNSUPPORTED;
  }
  const unsigned grid = (unsigned)mixed_max_tiles(a.n, a.nleaf);
  DRPT_CUDA(cudaFuncSetAttribute(k_leaf_mma<KP, SHAPE, FP8>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_leaf_mma<KP, SHAPE, FP8><<<grid, Cfg::threads, smem, s>>>(
      tmA, tmB, a.order, a.nrm, a.scl, a.tiles, a.n_tiles, kb, a.tree, a.cand_idx, a.cand_dist, a.tree_idx, a.tree_dist, a.err);
  DRPT_LAUNCH_CHECK();
  if (a.tree > 0) DRPT_TRY(launch_fold_lists(a, s));
  return DRPT_OK;
}

template <int KP, bool FP8>
drpt_status mma_shaped(const MixedTreeArgs &a, const CUtensorMap &tmA, int kb, cudaStream_t s) {
  if (kb <= 2) return mma_t<KP, 0, FP8>(a, tmA, kb, s);
  if constexpr (KP == 16)
    if (kb <= 4) return mma_t<KP, 1, FP8>(a, tmA, kb, s);
  if (wide_rows(kb, a.leaf_rows)) return mma_t<KP, 3, FP8>(a, tmA, kb, s);
  return mma_t<KP, 2, FP8>(a, tmA, kb, s);
}

template <int KP>
drpt_status mma_kp(const MixedTreeArgs &a, const CUtensorMap &tmA, int kb, cudaStream_t s) {
  return a.fp8 ? mma_shaped<KP, true>(a, tmA, kb, s) : mma_shaped<KP, false>(a, tmA, kb, s);
}

}  // namespace

// Padded row length of the mixed form's tensor-core operand: whole 128-byte
// K blocks (64 BF16 or 128 E4M3 values).
int mixed_d_pad(int d, int fp8) { return fp8 ? (d + 127) / 128 * 128 : (d + 63) / 64 * 64; }

static drpt_status stage_check(const LeafStageArgs &a) {
  if (a.d % 4 != 0 || a.d > 1024 || a.d_pad != mixed_d_pad(a.d, a.fp8)) {
    set_error("mixed mode needs d %% 4 == 0 and d <= 1024 (got %d)", a.d);
    return DRPT_ERR_UNSUPPORTED;
  }
  return DRPT_OK;
}

drpt_status launch_leaf_means(const LeafStageArgs &a, cudaStream_t s) {
  DRPT_TRY(stage_check(a));
  if (a.dtype == DRPT_DTYPE_U8) stage_d<uint8_t>(a, true, s);
  else stage_d<float>(a, true, s);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

drpt_status launch_leaf_stage(const LeafStageArgs &a, cudaStream_t s) {
  DRPT_TRY(stage_check(a));
  if (a.dtype == DRPT_DTYPE_U8) stage_d<uint8_t>(a, false, s);
  else stage_d<float>(a, false, s);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

int mixed_stage_trees(int64_t n, int d_pad, int fp8, int T) {
  // centred rows of as many trees as fit in 8 GiB
  const int64_t per_tree = n * d_pad * (fp8 ? 1 : 2);
  const int64_t fit = per_tree > 0 ? ((int64_t)8 << 30) / per_tree : T;
  return (int)std::max<int64_t>(1, std::min<int64_t>(T, fit));
}

drpt_status launch_leaf_mma(const MixedTreeArgs &a, cudaStream_t s) {
  const int esz = a.fp8 ? 1 : 2;
  if ((a.d_pad * esz) % 128 != 0 || a.d_pad > 1024) {
    set_error("mixed leaf kernel: padded dimension %d unsupported", a.d_pad);
    return DRPT_ERR_UNSUPPORTED;
  }
  CUtensorMap tmA;
  DRPT_TRY(make_tmap(&tmA, a.Xb, a.n, a.d_pad, kTM, a.fp8));
  const int kb = a.d_pad * esz / 128;
  if (a.kp == 16) return mma_kp<16>(a, tmA, kb, s);
  if (a.kp == 32) return mma_kp<32>(a, tmA, kb, s);
  set_error("mixed leaf kernel: %d candidates per tree unsupported (16 or 32)", a.kp);
  return DRPT_ERR_UNSUPPORTED;
}

int64_t mixed_max_tiles(int64_t n, int nleaf) { return ceil_div(n, kTM) + nleaf; }

drpt_status launch_tile_plan(const int32_t *goff, int64_t n, int T, int nleaf, int4 *tiles,
                             int32_t *n_tiles, cudaStream_t s) {
  k_tile_plan<<<(unsigned)T, 1024, 0, s>>>(goff, nleaf, mixed_max_tiles(n, nleaf), tiles, n_tiles);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

constexpr int64_t kFoldLanes = 1 << 18;  // points x entries
drpt_status launch_fold_lists(const MixedTreeArgs &a, cudaStream_t s) {
  if (a.kp != 16 && a.kp != 32) {
    set_error("fold: %d candidates per tree unsupported (16 or 32)", a.kp);
    return DRPT_ERR_UNSUPPORTED;
  }
  const bool lanes = a.n * a.kp <= kFoldLanes;
  const int threads = lanes ? 256 : kFoldThreads;
  const unsigned grid = (unsigned)ceil_div(lanes ? a.n * a.kp : a.n, threads);
  auto kern = a.kp == 16 ? (lanes ? k_fold_lanes<16> : k_fold_lists<16>)
                         : (lanes ? k_fold_lanes<32> : k_fold_lists<32>);
  kern<<<grid, threads, 0, s>>>(a.tree_dist, a.tree_idx, a.n, a.cand_dist, a.cand_idx);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

drpt_status launch_rerank(const void *X, int dtype, int d, const int32_t *visit, int64_t n,
                          const int32_t *cand, int K2, int k, int32_t *out_idx, float *out_dist,
                          cudaStream_t s) {
  if ((K2 != 16 && K2 != 32) || k > K2 || k <= 0) {
    set_error("re-rank: %d candidates for k = %d unsupported (16 or 32)", K2, k);
    return DRPT_ERR_UNSUPPORTED;
  }
  if (d % 4 != 0 || d > 1024) {
    set_error("re-rank needs d %% 4 == 0 and d <= 1024 (got %d)", d);
    return DRPT_ERR_UNSUPPORTED;
  }
  if (dtype == DRPT_DTYPE_U8)
    return K2 == 16 ? launch_rerank_d<uint8_t, 16>(X, d, visit, n, cand, k, out_idx, out_dist, s)
                    : launch_rerank_d<uint8_t, 32>(X, d, visit, n, cand, k, out_idx, out_dist, s);
  return K2 == 16 ? launch_rerank_d<float, 16>(X, d, visit, n, cand, k, out_idx, out_dist, s)
                  : launch_rerank_d<float, 32>(X, d, visit, n, cand, k, out_idx, out_dist, s);
}

}  // namespace drpt
