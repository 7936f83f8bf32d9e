// FP32 CUDA-core form of the whole-leaf brute force (DRPT_MODE_FP32_GRAM):
// the same trees, running list and exact FP32 re-rank as the mixed form, with
// the leaf Gram tiles computed in FP32 by fused multiply-adds on the CUDA
// cores (packed FP32x2 multiply-adds) instead of BF16 tiles on the tensor
// cores.  It is the fastest plain FP32 counterpart of the mixed form (the
// reference's own per-pair subtract / multiply / add sequence, kept bit for
// bit by the exact form's kernels, k_leaf_tri, k_leaf_tiles_exact and, above 32
// neighbours, k_leaf_knn, takes three FP32 operations per dimension and pair;
// this takes one).
//
//   k_row_norms   ||x||^2 of every row in FP32 (once per build)
//   k_leaf_f32    per CTA one 128-row tile of a global leaf against every
//                 128-column tile of the leaf: rows and columns gathered from
//                 X in 16-dimension chunks into shared memory (the next chunk
//                 loaded into registers while the current one is used), a
//                 16 x 8 register block of FFMA dot products per thread, then
//                 score ||y||^2 - 2 x.y per pair; a thread per row keeps the
//                 KP best (score, column) pairs, at the end of the row tile
//                 the tree's list of the row's point.  (The rows are not
//                 centred, so the scores are large next to the gaps between
//                 neighbours: the mixed form's packed keys, which give up the
//                 score's low 13 bits to the column, would rank them too
//                 coarsely.)
//
// The same tile loop with the reference's operation sequence per pair
// (subtract, multiply, add, each rounded on its own, then the square root)
// brute-forces the exact form's leaves of more than 128 points
// (k_leaf_tiles_exact).
//
// Reference: the leaf brute force MDRPT::calculate_nns (mdrpt.cpp:123-212)
// with MathOp::calculate_distance (math_operations.cpp:385-396).
#include "kernels.cuh"
#include "leaf_lists.cuh"
#include "sm100.cuh"
#include "warp_list.cuh"

namespace drpt {
namespace {

constexpr int kRows = 128;       // rows per tile
constexpr int kCols = 128;       // columns per tile
constexpr int kKc = 16;          // dimensions per staged chunk
constexpr int kPitch = kCols + 4;      // score-tile row pitch (words)
constexpr int kPool = kRows * kPitch;  // floats of the shared pool
static_assert(kKc == 16, "load_row16");
static_assert(2 * kKc * (kRows + kCols) <= kPool, "two buffers of staged chunks fit the pool");
template <int KP>
constexpr size_t f32_smem() {
  return sizeof(float) * (kPool + kCols + kRows * KP) + sizeof(int32_t) * kRows * KP;
}
constexpr int kMaxLeaf = 1 << 13;  // the mixed form's leaf limit

// Values c .. c + 7 of a row of which `left` remain (zero past them); `vec`:
// 16-byte (u8: 4-byte) pieces can be read.
template <typename T>
__device__ __forceinline__ void load_row8(const T *row, int left, int c, bool vec, float *v) {
  if (vec) {
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (h < left) {
        if constexpr (sizeof(T) == 1) {
          const uchar4 b = __ldg(reinterpret_cast<const uchar4 *>(row + c + h));
          q = make_float4(b.x, b.y, b.z, b.w);
        } else {
          q = __ldg(reinterpret_cast<const float4 *>(row + c + h));
        }
      }
      v[h] = q.x; v[h + 1] = q.y; v[h + 2] = q.z; v[h + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = e < left ? (float)__ldg(row + c + e) : 0.0f;
  }
}

// kKc (16) values c .. c + 15 of a row of which `left` remain, a multiple of 8
// (zero past them).  Bytes are read in pieces of `align` (16, 8 or 4; every
// row and piece starts on such a boundary): with 4-byte pieces the loads of a
// byte row take four times as many requests as they need (60,000 x 784, 4
// trees: 14.2 ms per build).
template <typename T>
__device__ __forceinline__ void load_row16(const T *row, int left, int c, int align, float *v) {
  if constexpr (sizeof(T) == 1) {
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (align == 16) {
      if (left > 0) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(row + c));
        w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (8 * h >= left) continue;
        if (align == 8) {
          const uint2 q = __ldg(reinterpret_cast<const uint2 *>(row + c) + h);
          w[2 * h] = q.x; w[2 * h + 1] = q.y;
        } else {
          w[2 * h] = __ldg(reinterpret_cast<const uint32_t *>(row + c) + 2 * h);
          w[2 * h + 1] = __ldg(reinterpret_cast<const uint32_t *>(row + c) + 2 * h + 1);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = (float)((w[e >> 2] >> (8 * (e & 3))) & 0xffu);
  } else {
    load_row8<T>(row, left, c, true, v);
    load_row8<T>(row, left - 8, c + 8, true, v + 8);
  }
}

// ||x||^2 per row: a warp per row, lanes over 4-value groups, a fixed
// butterfly for the lane sums.
template <typename T>
__global__ void __launch_bounds__(256) k_row_norms(const T *__restrict__ X, int64_t n, int d,
                                                   float *__restrict__ out) {
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const T *row = X + w * d;
  float s = 0.0f;
  for (int c = 4 * lane; c < d; c += 128)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float v = (float)row[c + e];
      s = fmaf(v, v, s);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
  if (lane == 0) out[w] = s;
}

// Ascending list of N (score, column) pairs <- the N smallest of it and (v, c)
// whose column is above every column in the list (the scan order): entry i becomes entry i - 1 where v < old entry i - 1, (v, c)
// where it falls between them, else stays; every entry from the old list at
// once, no chain through (v, c).  Equal scores keep the earlier column.
template <int N>
__device__ __forceinline__ void pair_shift_in(float *Lv, int32_t *Lc, float v, int32_t c) {
  bool below[N];
#pragma unroll
  for (int i = 0; i < N; ++i) below[i] = v < Lv[i];
#pragma unroll
  for (int i = N - 1; i > 0; --i) {
    Lv[i] = below[i - 1] ? Lv[i - 1] : (below[i] ? v : Lv[i]);
    Lc[i] = below[i - 1] ? Lc[i - 1] : (below[i] ? c : Lc[i]);
  }
  Lv[0] = below[0] ? v : Lv[0];
  Lc[0] = below[0] ? c : Lc[0];
}

// k_leaf_f32: one row tile per CTA of 128 threads, two CTAs per SM, so that
// one's selection runs under the other's products.  Thread (ty, tx) owns rows
// 32 g + 4 ty + i and columns 64 h + 4 tx + j (16 x 8): 24 values read from
// shared memory per 128 multiply-adds.  (A load returns 128 bytes per cycle
// and SM, broadcast or not: with 8 x 8 values per thread the loads take as
// long as the multiply-adds.)  Two rows per packed FP32x2 multiply-add, each
// dot product in its own FP32 sum in order of the dimensions.  In the
// selection a thread owns a row; its list lies in shared memory between tiles,
// which leaves its registers to the 128 sums.  262,144 x 128, 6 trees: 13.6 ->
// 10.8 ms of leaf kernels against one CTA of 256 threads with 8 x 8 values
// each (0.41 -> 0.51 of the FFMA rate); a warp per row in the selection, which
// needs fewer registers, took 19.3 ms.
constexpr int kF32Threads = 128;
template <typename T, int KP>
__global__ void __launch_bounds__(kF32Threads, 2) k_leaf_f32(
    const T *__restrict__ X, int d, const int32_t *__restrict__ order,
    const float *__restrict__ xnorm, const int4 *__restrict__ tiles,
    const int32_t *__restrict__ n_tiles, int tree, int32_t *__restrict__ run_idx,
    float *__restrict__ run_dist, int32_t *__restrict__ tree_idx, float *__restrict__ tree_dist,
    int align, int *err) {
  // pool: two buffers of staged chunks (rows, columns, dimension-major), then
  // the tile's scores; column norms; every row's list, entry-major
  extern __shared__ __align__(16) float smem[];
  float *pool = smem, *cnorm = pool + kPool;
  float *lv = cnorm + kCols;
  int32_t *lc = reinterpret_cast<int32_t *>(lv + KP * kRows);
  const int u = blockIdx.x;
  if (u >= *n_tiles) return;  // uniform for the whole block
  const int4 tile = __ldg(tiles + u);
  const int32_t lo = tile.x, m = tile.y;
  const int r0 = tile.z;
  if (m > kMaxLeaf) {
    if (threadIdx.x == 0) atomicOr(err, 2);
    empty_lists<KP>(order + lo + r0, min(kRows, m - r0), tree > 0 ? tree_idx : run_idx,
                    tree > 0 ? tree_dist : run_dist);
    return;
  }
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  auto As = [&](int b) { return pool + b * kKc * (kRows + kCols); };
  auto Bs = [&](int b) { return As(b) + kKc * kRows; };
  const float inf = __int_as_float(0x7f800000);
  // staging and selection: row (column) tid of the tiles
  const bool rvalid = r0 + tid < m;
  const int32_t arow = rvalid ? __ldg(order + lo + r0 + tid) : -1;
#pragma unroll
  for (int j = 0; j < KP; ++j) {
    lv[j * kRows + tid] = inf;
    lc[j * kRows + tid] = -1;
  }
  // later trees: candidates at or above the KP-th of the point's running
  // list (score = squared distance - ||x||^2) are never kept
  float thr0 = rvalid ? inf : -inf;
  if (tree > 0 && rvalid) thr0 = run_dist[(int64_t)arow * KP + KP - 1] - __ldg(xnorm + arow);
  float thr = thr0;
  // The next column tile's id, norm and first chunk are loaded while the
  // current tile is computed, so that no tile starts on global-memory latency
  // (the id, then the row it names).
  auto col_id = [&](int c0) { return c0 + tid < m ? __ldg(order + lo + c0 + tid) : -1; };
  float pa[kKc], pb[kKc];
  auto fetch = [&](int32_t bc, int k0) {
    load_row16<T>(X + (int64_t)max(arow, 0) * d, arow >= 0 ? d - k0 : 0, k0, align, pa);
    load_row16<T>(X + (int64_t)max(bc, 0) * d, bc >= 0 ? d - k0 : 0, k0, align, pb);
  };
  auto store = [&](int b) {
    float *A = As(b) + tid, *B = Bs(b) + tid;
#pragma unroll
    for (int e = 0; e < kKc; ++e) {
      A[e * kRows] = pa[e];
      B[e * kCols] = pb[e];
    }
  };
  int32_t bcol = col_id(0);
  float cn = bcol >= 0 ? __ldg(xnorm + bcol) : inf;
  fetch(bcol, 0);
  for (int c0 = 0; c0 < m; c0 += kCols) {
    const int32_t bnext = col_id(c0 + kCols);
    float2 acc[8][8];  // rows 32 (p / 2) + 4 ty + 2 (p % 2) + {0, 1}, columns 64 (j / 4) + 4 tx + j % 4
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[p][j] = make_float2(0.0f, 0.0f);
    __syncthreads();  // the previous tile's scores are no longer read
    cnorm[tid] = cn;
    store(0);
    __syncthreads();
    int cur = 0;
    for (int k0 = 0; k0 < d; k0 += kKc, cur ^= 1) {
      // in flight while this chunk is used: the next chunk, or the next
      // tile's first one
      const bool more = k0 + kKc < d;
      if (more) fetch(bcol, k0 + kKc);
      else if (c0 + kCols < m) fetch(bnext, 0);
      const float *A = As(cur) + 4 * ty, *B = Bs(cur) + 4 * tx;
#pragma unroll 4
      for (int kk = 0; kk < kKc; ++kk) {
        const float4 b0 = *reinterpret_cast<const float4 *>(B + kk * kCols);
        const float4 b1 = *reinterpret_cast<const float4 *>(B + kk * kCols + 64);
        const float y[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float4 a = *reinterpret_cast<const float4 *>(A + kk * kRows + 32 * g);
          const float2 x0 = make_float2(a.x, a.y), x1 = make_float2(a.z, a.w);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float2 yy = make_float2(y[j], y[j]);
            acc[2 * g][j] = sm100::fma2(x0, yy, acc[2 * g][j]);
            acc[2 * g + 1][j] = sm100::fma2(x1, yy, acc[2 * g + 1][j]);
          }
        }
      }
      // the other buffer was last read in the previous chunk, before the
      // barrier that ended it
      if (more) store(cur ^ 1);
      __syncthreads();
    }
    // scores ||y||^2 - 2 x.y (columns past the leaf: +inf)
    const float4 n0 = *reinterpret_cast<const float4 *>(cnorm + 4 * tx);
    const float4 n1 = *reinterpret_cast<const float4 *>(cnorm + 64 + 4 * tx);
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float *St = pool + (32 * (p >> 1) + 4 * ty + 2 * (p & 1) + h) * kPitch + 4 * tx;
        auto v = [&](int j) { return h ? acc[p][j].y : acc[p][j].x; };
        *reinterpret_cast<float4 *>(St) =
            make_float4(fmaf(-2.0f, v(0), n0.x), fmaf(-2.0f, v(1), n0.y), fmaf(-2.0f, v(2), n0.z),
                        fmaf(-2.0f, v(3), n0.w));
        *reinterpret_cast<float4 *>(St + 64) =
            make_float4(fmaf(-2.0f, v(4), n1.x), fmaf(-2.0f, v(5), n1.y), fmaf(-2.0f, v(6), n1.z),
                        fmaf(-2.0f, v(7), n1.w));
      }
    bcol = bnext;
    cn = bcol >= 0 ? __ldg(xnorm + bcol) : inf;
    __syncthreads();
    // a mask of the row's scores below the threshold at the tile's start (a
    // superset of those that enter the list), then its set bits in column
    // order, each tested again against the current threshold: the warp runs
    // the insertion as often as its busiest lane, not once per column where
    // any lane inserts
    const float *srow = pool + tid * kPitch;
    uint32_t pass[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 q = *reinterpret_cast<const float4 *>(srow + 32 * w + j);
        if (q.x < thr) pass[w] |= 1u << j;
        if (q.y < thr) pass[w] |= 2u << j;
        if (q.z < thr) pass[w] |= 4u << j;
        if (q.w < thr) pass[w] |= 8u << j;
      }
#pragma unroll
    for (int w = 0; w < 4; ++w)  // not the row's own column
      if ((r0 + tid - c0) >> 5 == w) pass[w] &= ~(1u << ((r0 + tid) & 31));
    if (__any_sync(kFull, pass[0] | pass[1] | pass[2] | pass[3])) {
      float tv[KP];
      int32_t tc[KP];
#pragma unroll
      for (int j = 0; j < KP; ++j) {
        tv[j] = lv[j * kRows + tid];
        tc[j] = lc[j * kRows + tid];
      }
      // the words one after the other through one copy of the insertion
      uint32_t bits = pass[0];
      int w = 0;
      for (;;) {
        while (!bits && w < 3) {
          ++w;
          bits = w == 1 ? pass[1] : (w == 2 ? pass[2] : pass[3]);
        }
        if (!bits) break;
        const int j = 32 * w + __ffs(bits) - 1;
        bits &= bits - 1;
        const float v = srow[j];
        if (v < thr) {  // (ties with the KP-th keep the earlier column)
          pair_shift_in<KP>(tv, tc, v, c0 + j);
          thr = fminf(thr0, tv[KP - 1]);
        }
      }
#pragma unroll
      for (int j = 0; j < KP; ++j) {
        lv[j * kRows + tid] = tv[j];
        lc[j * kRows + tid] = tc[j];
      }
    }
  }
  // the row's list: tree 0 straight into the running list, later trees into
  // the tree list (folded by k_fold_lists)
  if (rvalid) {
    const float nr = __ldg(xnorm + arow);
    const int64_t o = (int64_t)arow * KP;
    float *dd = (tree > 0 ? tree_dist : run_dist) + o;
    int32_t *di = (tree > 0 ? tree_idx : run_idx) + o;
#pragma unroll 4
    for (int j = 0; j < KP; ++j) {
      const int32_t c = lc[j * kRows + tid];
      di[j] = c >= 0 ? __ldg(order + lo + c) : -1;
      dd[j] = c >= 0 ? nr + lv[j * kRows + tid] : inf;
    }
  }
}

// k_leaf_tiles_exact: the exact form's leaves of more than `above` members.
// Block (tree, leaf) takes the leaf's 128-row tiles in turn against its
// 128-column tiles with the reference's operation sequence per pair; 256
// threads of 8 x 8 pairs, a warp per row keeps the k <= 32 best by (distance,
// id) of its lanes' columns, the lists in shared memory between tiles.
// 100,000 x 128 whole leaves of 1,024 (FP32 leaf form, 4 trees): build 19.5 ->
// 10.2 ms against 64 x 64 tiles with scalar operations and serial selection.
// Leaves just above 128 points pay for 256 x 256 pairs: of leaves of 128 on average,
// half of them above (131,072 points, 8 trees), 32 dimensions and 5 neighbours take
// 2.7 ms where those tiles took 2.1, 10 neighbours 3.1 and 3.3, 128 dimensions and
// 10 neighbours 5.8 and 6.2.
constexpr int kExactThreads = 256, kExactK = 32;
constexpr size_t kExactSmem =
    sizeof(float) * (kPool + kRows * kExactK) + sizeof(int32_t) * (kRows + kCols + kRows * kExactK);
template <typename T>
__global__ void __launch_bounds__(kExactThreads, 2) k_leaf_tiles_exact(LeafKnnArgs a, int above,
                                                                       bool vec) {
  extern __shared__ __align__(16) float smem[];
  float *pool = smem, *lv = pool + kPool;
  int32_t *lc = reinterpret_cast<int32_t *>(lv + kRows * kExactK);  // [row][entry]
  int32_t *rid = lc + kRows * kExactK, *cid = rid + kRows;
  const int t = blockIdx.x / a.n_final, f = blockIdx.x - t * a.n_final;
  const int32_t *off = a.final_off + (int64_t)t * (a.n_final + 1);
  const int32_t lo = off[f], m = off[f + 1] - lo;
  if (m <= above) return;
  const int32_t *ord = a.final_order + (int64_t)t * a.n + lo;
  const T *X = (const T *)a.X;
  const int d = a.d, k = a.k;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int warp = tid >> 5, lane = tid & 31;
  const float inf = __int_as_float(0x7f800000);
  auto As = [&](int b) { return pool + b * kKc * (kRows + kCols); };
  auto Bs = [&](int b) { return As(b) + kKc * kRows; };
  // staging: row and column sr of the tiles, 8 dimensions from sk
  const int sr = tid & (kRows - 1), sk = (tid >> 7) * 8;
  for (int r0 = 0; r0 < m; r0 += kRows) {
    const int rows = min(kRows, m - r0);
    const int32_t arow = sr < rows ? __ldg(ord + r0 + sr) : -1;
    __syncthreads();  // the previous row tile's ids and lists are written out
    if (tid < kRows) rid[tid] = arow;
    for (int i = tid; i < kRows * kExactK; i += kExactThreads) {
      lv[i] = inf;
      lc[i] = -1;
    }
    auto col_id = [&](int c0) { return c0 + sr < m ? __ldg(ord + c0 + sr) : -1; };
    float pa[8], pb[8];
    auto fetch = [&](int32_t bc, int k0) {
      load_row8<T>(X + (int64_t)max(arow, 0) * d, arow >= 0 ? d - (k0 + sk) : 0, k0 + sk, vec, pa);
      load_row8<T>(X + (int64_t)max(bc, 0) * d, bc >= 0 ? d - (k0 + sk) : 0, k0 + sk, vec, pb);
    };
    auto store = [&](int b) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        As(b)[(sk + e) * kRows + sr] = pa[e];
        Bs(b)[(sk + e) * kCols + sr] = pb[e];
      }
    };
    int32_t bcol = col_id(0);
    fetch(bcol, 0);
    for (int c0 = 0; c0 < m; c0 += kCols) {
      const int32_t bnext = col_id(c0 + kCols);
      float2 acc[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
      __syncthreads();  // the previous tile's distances are no longer read
      if (tid < kCols) cid[tid] = bcol;
      store(0);
      __syncthreads();
      int cur = 0;
      for (int k0 = 0; k0 < d; k0 += kKc, cur ^= 1) {
        const bool more = k0 + kKc < d;
        if (more) fetch(bcol, k0 + kKc);
        const float *A = As(cur) + 4 * ty, *B = Bs(cur) + 4 * tx;
#pragma unroll 4
        for (int kk = 0; kk < kKc; ++kk) {
          const float4 b0 = *reinterpret_cast<const float4 *>(B + kk * kCols);
          const float4 b1 = *reinterpret_cast<const float4 *>(B + kk * kCols + 64);
          const float y[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const float4 q = *reinterpret_cast<const float4 *>(A + kk * kRows + 64 * g);
            const float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float d0 = __fsub_rn(y[2 * j], x[i]), d1 = __fsub_rn(y[2 * j + 1], x[i]);
                acc[4 * g + i][j] = sm100::add2(
                    acc[4 * g + i][j], make_float2(__fmul_rn(d0, d0), __fmul_rn(d1, d1)));
              }
          }
        }
        if (more) store(cur ^ 1);
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float *St = pool + ((i < 4 ? 0 : 60) + 4 * ty + i) * kPitch + 4 * tx;
        *reinterpret_cast<float4 *>(St) =
            make_float4(__fsqrt_rn(acc[i][0].x), __fsqrt_rn(acc[i][0].y),
                        __fsqrt_rn(acc[i][1].x), __fsqrt_rn(acc[i][1].y));
        *reinterpret_cast<float4 *>(St + 64) =
            make_float4(__fsqrt_rn(acc[i][2].x), __fsqrt_rn(acc[i][2].y),
                        __fsqrt_rn(acc[i][3].x), __fsqrt_rn(acc[i][3].y));
      }
      bcol = bnext;
      if (c0 + kCols < m) fetch(bcol, 0);  // the next tile's first chunk
      __syncthreads();
      // warp w takes rows 16 w .., lane l the columns l + 32 h
      int32_t ids[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) ids[h] = cid[32 * h + lane];
      for (int r = 16 * warp; r < min(16 * warp + 16, rows); ++r) {
        const float *St = pool + r * kPitch;
        float ld = lv[r * kExactK + lane];
        int32_t li = lc[r * kExactK + lane];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const float v = St[32 * h + lane];
          const bool own = c0 + 32 * h + lane == r0 + r;
          warp_take(ld, li, v, own ? -1 : ids[h], k, lane);
        }
        lv[r * kExactK + lane] = ld;
        lc[r * kExactK + lane] = li;
      }
    }
    for (int r = 16 * warp; r < min(16 * warp + 16, rows); ++r)  // the warp's own rows
      if (lane < k) {
        const int64_t o = ((int64_t)rid[r] * a.T + t) * k + lane;
        a.cand_idx[o] = lc[r * kExactK + lane];
        a.cand_dist[o] = lv[r * kExactK + lane];
      }
  }
}

template <typename T, int KP>
drpt_status f32_launch(const MixedTreeArgs &a, const float *xnorm, unsigned grid, cudaStream_t s) {
  DRPT_CUDA(cudaFuncSetAttribute(k_leaf_f32<T, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)f32_smem<KP>()));
  const int step = sizeof(T) == 1 && a.d % 16 == 0 ? 16 : 8;
  const int align = (uintptr_t)a.X % step == 0 ? step : ((uintptr_t)a.X % 8 == 0 ? 8 : 4);
  k_leaf_f32<T, KP><<<grid, kF32Threads, f32_smem<KP>(), s>>>(
      (const T *)a.X, a.d, a.order, xnorm, a.tiles, a.n_tiles, a.tree, a.cand_idx, a.cand_dist,
      a.tree_idx, a.tree_dist, align, a.err);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

template <typename T>
drpt_status tiles_exact(const LeafKnnArgs &a, int above, unsigned blocks, cudaStream_t s) {
  // rows start on 16-byte (u8: 4-byte) boundaries
  const bool vec = a.d % 4 == 0 && (uintptr_t)a.X % (4 * sizeof(T)) == 0;
  DRPT_CUDA(cudaFuncSetAttribute(k_leaf_tiles_exact<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kExactSmem));
  k_leaf_tiles_exact<T><<<blocks, kExactThreads, kExactSmem, s>>>(a, above, vec);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

}  // namespace

drpt_status launch_leaf_tiles_exact(const LeafKnnArgs &a, int above, cudaStream_t s) {
  const unsigned blocks = (unsigned)((int64_t)a.T * a.n_final);
  return a.dtype == DRPT_DTYPE_U8 ? tiles_exact<uint8_t>(a, above, blocks, s)
                                  : tiles_exact<float>(a, above, blocks, s);
}

drpt_status launch_row_norms(const void *X, int dtype, int64_t n, int d, float *out,
                             cudaStream_t s) {
  const unsigned grid = (unsigned)ceil_div(n * 32, 256);
  if (dtype == DRPT_DTYPE_U8)
    k_row_norms<uint8_t><<<grid, 256, 0, s>>>((const uint8_t *)X, n, d, out);
  else
    k_row_norms<float><<<grid, 256, 0, s>>>((const float *)X, n, d, out);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

drpt_status launch_leaf_f32(const MixedTreeArgs &a, const float *xnorm, cudaStream_t s) {
  if (a.d % 8 != 0) {
    set_error("FP32 Gram leaf kernel: d %% 8 == 0 needed (got %d)", a.d);
    return DRPT_ERR_UNSUPPORTED;
  }
  const unsigned grid = (unsigned)mixed_max_tiles(a.n, a.nleaf);
  drpt_status st;
  if (a.kp == 16)
    st = a.dtype == DRPT_DTYPE_U8 ? f32_launch<uint8_t, 16>(a, xnorm, grid, s)
                                  : f32_launch<float, 16>(a, xnorm, grid, s);
  else if (a.kp == 32)
    st = a.dtype == DRPT_DTYPE_U8 ? f32_launch<uint8_t, 32>(a, xnorm, grid, s)
                                  : f32_launch<float, 32>(a, xnorm, grid, s);
  else {
    set_error("FP32 Gram leaf kernel: %d candidates per tree unsupported (16 or 32)", a.kp);
    return DRPT_ERR_UNSUPPORTED;
  }
  DRPT_TRY(st);
  DRPT_LAUNCH_CHECK();
  if (a.tree > 0) DRPT_TRY(launch_fold_lists(a, s));
  return DRPT_OK;
}

}  // namespace drpt
