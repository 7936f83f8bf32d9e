// K1 -- sparse random projection P = X.B (math_operations.cpp:15-46 through
// an ordered sgemm).  Each point row is read once, coalesced, into shared
// memory; each output column is written once, coalesced.
//
// Per output element the sum runs over the nonzeros of B's column in
// ascending k with one rounded multiply and one rounded add per term
// (__fmul_rn / __fadd_rn, never contracted).  Zero entries of B are skipped:
// for finite inputs they add +-0 to an accumulator that starts at +0 and so
// never changes it, which keeps P bit-identical to the sequential sum over
// all d terms.
#include <type_traits>

#include "kernels.cuh"

namespace drpt {
namespace {

template <typename T>
__device__ __forceinline__ float to_f(T v) { return (float)v; }

// Four consecutive elements (16-byte or 4-byte aligned) as floats.
__device__ __forceinline__ float4 load4v(const float *p) {
  return __ldg(reinterpret_cast<const float4 *>(p));
}
__device__ __forceinline__ float4 load4v(const uint8_t *p) {
  const uchar4 q = __ldg(reinterpret_cast<const uchar4 *>(p));
  return make_float4(q.x, q.y, q.z, q.w);
}

// Block: PT consecutive points (or the block table's entry: first point,
// points, column set), staged as floats one dimension after the other; four
// points share 16 bytes, and quad g of dimension k stands at g ^ (k / 4 % 8), so
// that a warp's load of eight quads of four rows (128 consecutive bytes a row) is
// stored on all banks.  Eight loads in flight.  Products: a lane has four
// points, PT / 4 lanes a column, so a warp works on 128 / PT columns at a time
// and a step of four nonzeros has four independent 16-byte reads; columns of
// fewer nonzeros wait for the longest of the warp.  Instructions bound it (13 per
// nonzero and 128 points at best; a value read by a lane is 128 bytes a warp and
// cycle).  Against a lane per point and a warp per column, rows staged as they
// are: 1M x 128, 60 columns 277 -> 226 us, 250,000 x 256 146 -> 111, 60,000 x 784
// (8 bit) 112 -> 95, 500,000 x 960 3.48 -> 1.85 ms (25 of 32 lanes had a point
// there); 64 x 96 batches 570 -> 575.
template <typename T, int PT, int THREADS>
__global__ void __launch_bounds__(THREADS) k_project(const T *__restrict__ X, int64_t n, int d,
                                                 CscDev csc, float *__restrict__ P, bool quads,
                                                 bool vec_out) {
  constexpr uint32_t kRow = 4 * PT;                   // bytes of a dimension
  static_assert(PT >= 8, "quads to exchange");
  constexpr uint32_t kSwap = 16 * (PT >= 32 ? 7 : PT / 4 - 1);  // its quads' exchange
  extern __shared__ __align__(16) uint8_t xs[];  // d x kRow
  // byte at which dimension k has the quad of points that starts at byte q16
  const auto place = [](uint32_t k, uint32_t q16) { return k * kRow + (q16 ^ ((4 * k) & kSwap)); };
  int64_t p0 = (int64_t)blockIdx.x * PT;
  int np = (int)min64(PT, n - p0);
  if (csc.blocks) {
    const int32_t *b = csc.blocks + 3 * (int64_t)blockIdx.x;
    p0 = b[0];
    np = b[1];
    csc.colptr += (int64_t)b[2] * (csc.ncols + 1);
  }
  if (np <= 0) return;  // uniform for the whole block
  const T *src = X + p0 * d;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  if (quads) {
    constexpr int kBatch = 8, kRowSets = PT / 4;
    const int q4 = d >> 2, tasks = kRowSets * ((q4 + 7) >> 3);
    const int lr = lane >> 3, lq = lane & 7;
    for (int t0 = warp; t0 < tasks; t0 += kBatch * warps) {
      float4 v[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int t = t0 + i * warps, r = 4 * (t % kRowSets) + lr, q = 8 * (t / kRowSets) + lq;
        if (r < np && q < q4) v[i] = load4v(src + (int64_t)r * d + 4 * q);
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int t = t0 + i * warps, r = 4 * (t % kRowSets) + lr, q = 8 * (t / kRowSets) + lq;
        if (r < np && q < q4) {
          float *dst = reinterpret_cast<float *>(xs + place(4 * q, 4 * (r & ~3))) + lr;
          dst[0] = v[i].x;
          dst[PT] = v[i].y;
          dst[2 * PT] = v[i].z;
          dst[3 * PT] = v[i].w;
        }
      }
    }
  } else {
    // consecutive threads read consecutive elements of a row
    const int total = np * d;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int r = e / d, c = e - r * d;
      reinterpret_cast<float *>(xs + place(c, 4 * (r & ~3)))[r & 3] = to_f(src[e]);
    }
  }
  __syncthreads();
  // points past the block's are summed over what lies there and not written
  constexpr int kLanes = PT / 4, kCols = 32 / kLanes;
  const int pt = 4 * (lane % kLanes);
  // (lanes past the last column repeat it and write nothing)
  int e0 = 0, e1 = 0;
  const auto bounds = [&](int c) {
    const int col = min(c + lane / kLanes, csc.ncols - 1);
    e0 = __ldg(csc.colptr + col);
    e1 = __ldg(csc.colptr + col + 1);
  };
  bounds(kCols * warp);
  for (int c0 = kCols * warp; c0 < csc.ncols; c0 += kCols * warps) {
    const int col = c0 + lane / kLanes, len = e1 - e0;
    const int32_t *row = csc.row + e0;
    const float *val = csc.val + e0;
    const int least = kCols == 1 ? len : __reduce_min_sync(0xffffffffu, len);
    const int most = kCols == 1 ? len : __reduce_max_sync(0xffffffffu, len);
    bounds(c0 + kCols * warps);  // the next columns'
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const auto term = [&](const float4 &x, float b) {
      acc.x = __fadd_rn(acc.x, __fmul_rn(x.x, b));
      acc.y = __fadd_rn(acc.y, __fmul_rn(x.y, b));
      acc.z = __fadd_rn(acc.z, __fmul_rn(x.z, b));
      acc.w = __fadd_rn(acc.w, __fmul_rn(x.w, b));
    };
    const auto points = [&](int k) {
      return *reinterpret_cast<const float4 *>(xs + place(k, 4 * pt));
    };
    constexpr int kStep = 4;
    const auto step = [&](int s, auto all) {  // all: the warp's columns have these nonzeros
      int k[kStep];
      float b[kStep];
      float4 x[kStep];
#pragma unroll
      for (int i = 0; i < kStep; ++i) {
        const bool live = all.value || s + i < len;
        k[i] = live ? __ldg(row + s + i) : 0;
        b[i] = live ? __ldg(val + s + i) : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < kStep; ++i) x[i] = points(k[i]);
#pragma unroll
      for (int i = 0; i < kStep; ++i)
        if (all.value || s + i < len) term(x[i], b[i]);
    };
    int s = 0;
    for (; s + kStep <= least; s += kStep) step(s, std::true_type());
    if constexpr (kCols == 1) {
      for (; s < len; ++s) term(points(__ldg(row + s)), __ldg(val + s));
    } else {
      for (; s < most; s += kStep) step(s, std::false_type());
    }
    if (col >= csc.ncols) continue;
    float *out = P + (int64_t)col * n + p0 + pt;
    if (vec_out && p0 % 4 == 0 && pt + 4 <= np) {
      *reinterpret_cast<float4 *>(out) = acc;
    } else {
      if (pt < np) out[0] = acc.x;
      if (pt + 1 < np) out[1] = acc.y;
      if (pt + 2 < np) out[2] = acc.z;
      if (pt + 3 < np) out[3] = acc.w;
    }
  }
}

constexpr size_t kHalfSmem = 113 * 1024;  // two blocks per SM

size_t project_smem(int pts, int d) { return (size_t)d * pts * sizeof(float); }

template <typename T>
void project_t(const T *X, int64_t n, int d, const CscDev &csc, float *P, int pts, unsigned grid,
               cudaStream_t s) {
  const size_t smem = project_smem(pts, d);
  const bool quads = d % 4 == 0 && (uintptr_t)X % (4 * sizeof(T)) == 0;
  const bool vec_out = n % 4 == 0 && (uintptr_t)P % 16 == 0;
  auto launch = [&](auto kern, int threads) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<grid, threads, smem, s>>>(X, n, d, csc, P, quads, vec_out);
  };
  // a block that has the SM for itself takes 1,024 threads (500,000 x 960: 2.06 ->
  // 1.85 ms against 512).  The bound of k_project<T, 64> is above its threads:
  // with 256 the compiler takes 57 registers and 157 us for 250,000 x 256, not 76
  // and 112.
  if (pts == 128) launch(k_project<T, 128, 256>, 256);
  else if (pts == 64) launch(k_project<T, 64, 512>, 256);
  else if (smem <= kHalfSmem) launch(k_project<T, 32, 256>, 256);
  else if (pts == 32) launch(k_project<T, 32, 1024>, 1024);
  else if (pts == 16) launch(k_project<T, 16, 1024>, 1024);
  else launch(k_project<T, 8, 1024>, 1024);
}

}  // namespace

// 128 or 64 points while two such blocks fit on an SM, then 32 or what one
// block holds: 8 at the largest d that launch_project takes.
int project_points_per_block(int d) {
  for (int pts = 128; pts > 32; pts /= 2)
    if (project_smem(pts, d) <= kHalfSmem) return pts;
  int pts = 32;
  while (pts > 8 && project_smem(pts, d) > 227 * 1024) pts /= 2;
  return pts;
}

drpt_status launch_project(const void *X, int dtype, int64_t n, int d, const CscDev &csc,
                           float *P, cudaStream_t s) {
  if (n <= 0 || csc.ncols <= 0) return DRPT_OK;
  if ((size_t)8 * (d + 1) * sizeof(float) > 227 * 1024) {
    set_error("projection: d = %d too large for one staged row block", d);
    return DRPT_ERR_UNSUPPORTED;
  }
  int pts = project_points_per_block(d);
  // few points: smaller blocks, down to 32, until every SM has one
  while (!csc.blocks && pts > 32 && ceil_div(n, pts) < device_sm_count()) pts /= 2;
  const unsigned grid = csc.blocks ? (unsigned)csc.nblocks : (unsigned)ceil_div(n, pts);
  if (dtype == DRPT_DTYPE_U8)
    project_t(static_cast<const uint8_t *>(X), n, d, csc, P, pts, grid, s);
  else
    project_t(static_cast<const float *>(X), n, d, csc, P, pts, grid, s);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

}  // namespace drpt
