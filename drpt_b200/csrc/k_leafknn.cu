// K6 -- exact FP32 brute force inside every final leaf (MDRPT::calculate_nns,
// mdrpt.cpp:123-212, with MathOp::calculate_distance, math_operations.cpp:
// 385-396).
//
// One thread block per (tree, final leaf).  Per pair the distance chain is
// acc = acc + (q_i - p_i)^2 for i ascending, each subtract, multiply and add
// rounded on its own, then sqrt -- the reference's saxpy (-1) + snrm2
// sequence, so every distance is bit-identical to the reference's (a
// zero-padded dimension adds (0 - 0)^2 = +0, which leaves a non-negative sum
// unchanged; the two orders of a pair give the same distance).
//
//   k_leaf_tri          k <= 32, leaves of up to 128 points: each pair once
//   k_leaf_tiles_exact  k <= 32, larger leaves (k_fp32gram.cu)
//   k_leaf_knn          k > 32: 64 x 64 tiles of all pairs, one thread per row
//                       folding the tile's candidates into its list.  (Leaves of
//                       65 to 128 points in one 128 x 128 tile are slower, fewer
//                       CTAs fit an SM: 100,000 x 128, 8 trees, leaves of about
//                       98, 33 neighbours 13.4 ms of leaf kernels, 7.6 so; 64
//                       neighbours 22.3 and 15.9.)
//
// Output: for point p and tree t, cand[(p*T + t)*k + j], j < k, sorted by
// (distance, index), the point itself excluded; slots beyond the leaf size
// hold index -1 and distance +inf.
#include "kernels.cuh"
#include "sm100.cuh"
#include "warp_list.cuh"

namespace drpt {
namespace {

constexpr int kThreads = 256;
constexpr int kTile = 64;              // k_leaf_knn: rows and columns of a tile
constexpr int kChunk = 32;             // dimensions staged per step
constexpr int kLd = kChunk + 1;        // padded row stride in shared memory
constexpr int kTriThreads = 160;       // k_leaf_tri: threads, dimensions staged per step
constexpr int kTriKc = 32;

template <typename T>
__device__ __forceinline__ void stage_rows(float *dst, const T *__restrict__ X, int d,
                                           const int32_t *ids, int rows, int k0) {
  for (int e = threadIdx.x; e < kTile * kChunk; e += kThreads) {
    const int r = e / kChunk, kk = e - r * kChunk;
    float v = 0.0f;
    if (r < rows && k0 + kk < d) v = (float)X[(int64_t)ids[r] * d + k0 + kk];
    dst[r * kLd + kk] = v;
  }
}

constexpr size_t leaf_smem(int k) {
  return sizeof(float) * (2 * kTile * kLd + kTile * (kTile + 1)) +
         (sizeof(float) + sizeof(int32_t)) * kTile * (k + 1) + sizeof(int32_t) * 2 * kTile;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_leaf_knn(LeafKnnArgs a) {
  constexpr int TM = kTile, MT = TM / 16;
  extern __shared__ float smem[];
  float *xr = smem;                          // TM x kLd
  float *xc = xr + TM * kLd;                 // TM x kLd
  float *dt = xc + TM * kLd;                 // TM x (TM + 1)
  float *topd = dt + TM * (TM + 1);          // TM x (k + 1)
  int32_t *topi = (int32_t *)(topd + TM * (a.k + 1));
  int32_t *rid = topi + TM * (a.k + 1);      // TM
  int32_t *cid = rid + TM;                   // TM

  const int t = blockIdx.x / a.n_final, f = blockIdx.x - t * a.n_final;
  const int32_t *off = a.final_off + (int64_t)t * (a.n_final + 1);
  const int32_t b = off[f], m = off[f + 1] - b;
  const int32_t *members = a.final_order + (int64_t)t * a.n + b;
  const T *X = (const T *)a.X;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int kp1 = a.k + 1;
  const float inf = __int_as_float(0x7f800000);

  for (int r0 = 0; r0 < m; r0 += TM) {
    const int rows = min(TM, m - r0);
    for (int i = threadIdx.x; i < TM * kp1; i += kThreads) {
      topd[i] = inf;
      topi[i] = INT32_MAX;
    }
    if (threadIdx.x < TM) rid[threadIdx.x] = threadIdx.x < rows ? members[r0 + threadIdx.x] : -1;
    for (int c0 = 0; c0 < m; c0 += TM) {
      const int cols = min(TM, m - c0);
      const bool same = (c0 == r0);
      if (threadIdx.x < TM) cid[threadIdx.x] = threadIdx.x < cols ? members[c0 + threadIdx.x] : -1;
      __syncthreads();
      float acc[MT][MT];
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < MT; ++j) acc[i][j] = 0.0f;
      const float *xcol = same ? xr : xc;
      for (int k0 = 0; k0 < a.d; k0 += kChunk) {
        stage_rows(xr, X, a.d, rid, rows, k0);
        if (!same) stage_rows(xc, X, a.d, cid, cols, k0);
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < kChunk; ++kk) {
          float av[MT], bv[MT];
#pragma unroll
          for (int i = 0; i < MT; ++i) av[i] = xr[(ty + 16 * i) * kLd + kk];
#pragma unroll
          for (int j = 0; j < MT; ++j) bv[j] = xcol[(tx + 16 * j) * kLd + kk];
#pragma unroll
          for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < MT; ++j) {
              const float df = __fsub_rn(bv[j], av[i]);
              acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(df, df));
            }
        }
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < MT; ++j) dt[(ty + 16 * i) * (TM + 1) + tx + 16 * j] = __fsqrt_rn(acc[i][j]);
      __syncthreads();
      if (threadIdx.x < rows) {
        const int r = threadIdx.x;
        const int32_t p = rid[r];
        float *ld = topd + r * kp1;
        int32_t *li = topi + r * kp1;
        float wd = ld[a.k - 1];
        int32_t wi = li[a.k - 1];
        for (int c = 0; c < cols; ++c) {
          const int32_t q = cid[c];
          const float dv = dt[r * (TM + 1) + c];
          if (q == p || !(dv < wd || (dv == wd && q < wi))) continue;
          int j = a.k - 1;
          while (j > 0 && (dv < ld[j - 1] || (dv == ld[j - 1] && q < li[j - 1]))) {
            ld[j] = ld[j - 1];
            li[j] = li[j - 1];
            --j;
          }
          ld[j] = dv;
          li[j] = q;
          wd = ld[a.k - 1];
          wi = li[a.k - 1];
        }
      }
      __syncthreads();
    }
    if (threadIdx.x < rows) {
      const int r = threadIdx.x;
      const int64_t o = ((int64_t)rid[r] * a.T + t) * a.k;
      for (int j = 0; j < a.k; ++j) {
        const bool have = topi[r * kp1 + j] != INT32_MAX;
        a.cand_idx[o + j] = have ? topi[r * kp1 + j] : -1;
        a.cand_dist[o + j] = have ? topd[r * kp1 + j] : inf;
      }
    }
    __syncthreads();
  }
}

// k_leaf_tri: leaves of `above` < m <= MAXM points.  The m x m distances are
// symmetric, so only the 4 x 4 blocks on and above the diagonal are computed
// (numbered along the block columns), P of them per thread: block b of the
// ceil(m/4) (ceil(m/4) + 1) / 2 goes to thread b % NT.  The rows are staged in
// kTriKc-dimension chunks, dimension major, by steps that several resident CTAs
// overlap.  The distances then lie in shared memory
// (over the chunk), and a warp per row selects: the first 32 columns sorted
// over the lanes, later ones inserted below the k-th.
//
// FP32 issue bounds it: three operations per dimension and pair.  131,072 x
// 128, 16 trees (leaves of about 64): 7.9 -> 2.4 ms against 64 x 64 and 128 x
// 128 tiles of all pairs with a serial selection by one thread per row.  (With
// the rows also stored negated and doubled for a packed subtraction the loads
// from shared memory bound it: 2.8 ms.)
template <typename T, int MAXM, int P>
__global__ void __launch_bounds__(kTriThreads) k_leaf_tri(LeafKnnArgs a, int above, bool vec) {
  constexpr int NT = kTriThreads, kPitch = MAXM + 4;
  static_assert(P * NT >= (MAXM / 4) * (MAXM / 4 + 1) / 2, "every block has a thread");
  extern __shared__ __align__(16) float smem[];
  float *val = smem;  // [kTriKc][MAXM]
  float *dt = smem;   // [MAXM][kPitch]
  __shared__ int32_t ids[MAXM];
  const int t = blockIdx.x / a.n_final, f = blockIdx.x - t * a.n_final;
  const int32_t *off = a.final_off + (int64_t)t * (a.n_final + 1);
  const int32_t lo = off[f], m = off[f + 1] - lo;
  if (m <= above || m > MAXM) return;
  const int32_t *members = a.final_order + (int64_t)t * a.n + lo;
  const T *X = (const T *)a.X;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = (m + 3) >> 2, m4 = 4 * nb, nt = nb * (nb + 1) / 2;
  for (int i = tid; i < m4; i += NT) ids[i] = i < m ? __ldg(members + i) : -1;
  int bi[P], bj[P];  // block row <= block column
#pragma unroll
  for (int p = 0; p < P; ++p) {
    // column j holds the blocks j (j + 1) / 2 .. j (j + 1) / 2 + j
    const int b = min(tid + p * NT, nt - 1);
    int j = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);
    j += (j + 1) * (j + 2) / 2 <= b;
    j -= j * (j + 1) / 2 > b;
    bj[p] = 4 * j;
    bi[p] = 4 * (b - j * (j + 1) / 2);
  }
  float2 acc[P][4][2];
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[p][i][0] = acc[p][i][1] = make_float2(0.0f, 0.0f);
  __syncthreads();
  for (int k0 = 0; k0 < a.d; k0 += kTriKc) {
    // piece e: row e % m4, dimensions k0 + 4 (e / m4) .. + 3
    for (int e = tid; e < m4 * (kTriKc / 4); e += NT) {
      const int c = 4 * (e / m4), r = e - (c >> 2) * m4;
      const int32_t id = ids[r];
      const int left = id >= 0 ? a.d - (k0 + c) : 0;
      const T *src = X + (int64_t)max(id, 0) * a.d + k0 + c;
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (vec) {  // d % 4 == 0
        if (left > 0) {
          if constexpr (sizeof(T) == 1) {
            const uchar4 q = __ldg(reinterpret_cast<const uchar4 *>(src));
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
          } else {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(src));
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < left) v[i] = (float)__ldg(src + i);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) val[(c + i) * MAXM + r] = v[i];
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < P; ++p) {
      if (warp * 32 + p * NT >= nt) break;  // warp-uniform
      const float *x = val + bi[p], *y = val + bj[p];
#pragma unroll 4
      for (int kk = 0; kk < kTriKc; ++kk) {
        const float4 b = *reinterpret_cast<const float4 *>(y + kk * MAXM);
        const float4 q = *reinterpret_cast<const float4 *>(x + kk * MAXM);
        const float xs[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // two rounded subtractions and products, one packed addition
          float d0 = __fsub_rn(b.x, xs[i]), d1 = __fsub_rn(b.y, xs[i]);
          acc[p][i][0] =
              sm100::add2(acc[p][i][0], make_float2(__fmul_rn(d0, d0), __fmul_rn(d1, d1)));
          d0 = __fsub_rn(b.z, xs[i]);
          d1 = __fsub_rn(b.w, xs[i]);
          acc[p][i][1] =
              sm100::add2(acc[p][i][1], make_float2(__fmul_rn(d0, d0), __fmul_rn(d1, d1)));
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if (tid + p * NT < nt) {
      float4 q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[i] = make_float4(__fsqrt_rn(acc[p][i][0].x), __fsqrt_rn(acc[p][i][0].y),
                           __fsqrt_rn(acc[p][i][1].x), __fsqrt_rn(acc[p][i][1].y));
        *reinterpret_cast<float4 *>(dt + (bi[p] + i) * kPitch + bj[p]) = q[i];
      }
      float *m0 = dt + bj[p] * kPitch + bi[p];  // the mirrored block
      *reinterpret_cast<float4 *>(m0) = make_float4(q[0].x, q[1].x, q[2].x, q[3].x);
      *reinterpret_cast<float4 *>(m0 + kPitch) = make_float4(q[0].y, q[1].y, q[2].y, q[3].y);
      *reinterpret_cast<float4 *>(m0 + 2 * kPitch) = make_float4(q[0].z, q[1].z, q[2].z, q[3].z);
      *reinterpret_cast<float4 *>(m0 + 3 * kPitch) = make_float4(q[0].w, q[1].w, q[2].w, q[3].w);
    }
  }
  __syncthreads();
  const float inf = __int_as_float(0x7f800000);
  for (int r = warp; r < m; r += NT / 32) {
    const float *row = dt + r * kPitch;
    auto entry = [&](int c, float *d, int32_t *id) {
      const bool in = c < m && c != r;
      *d = in ? row[c] : inf;
      *id = in ? ids[c] : -1;
      if (!(*d <= inf)) *id = -1;  // a NaN distance enters no list
    };
    float ld, cd;
    int32_t li, ci;
    entry(lane, &ld, &li);
    if (li < 0) ld = inf;
    warp_sort32(ld, li, lane);
    for (int c0 = 32; c0 < m; c0 += 32) {
      entry(c0 + lane, &cd, &ci);
      warp_take(ld, li, cd, ci, a.k, lane);
    }
    if (lane < a.k) {
      const int64_t o = ((int64_t)ids[r] * a.T + t) * a.k + lane;
      a.cand_idx[o] = li;
      a.cand_dist[o] = li >= 0 ? ld : inf;
    }
  }
}

template <typename T, int MAXM, int P>
drpt_status launch_tri(const LeafKnnArgs &a, int above, bool vec, unsigned blocks,
                       cudaStream_t s) {
  constexpr size_t smem =
      sizeof(float) * MAXM * (kTriKc > MAXM + 4 ? kTriKc : MAXM + 4);
  DRPT_CUDA(cudaFuncSetAttribute(k_leaf_tri<T, MAXM, P>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_leaf_tri<T, MAXM, P><<<blocks, kTriThreads, smem, s>>>(a, above, vec);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

// Leaf classes of 1, 2 and 4 blocks per thread (17, 24 and 32 block columns);
// every launch covers all leaves and returns at once for the other classes.
template <typename T>
drpt_status launch_tris(const LeafKnnArgs &a, unsigned blocks, cudaStream_t s) {
  // rows start on 16-byte (u8: 4-byte) boundaries
  const bool vec = a.d % 4 == 0 && (uintptr_t)a.X % (4 * sizeof(T)) == 0;
  DRPT_TRY((launch_tri<T, 68, 1>(a, 0, vec, blocks, s)));
  DRPT_TRY((launch_tri<T, 96, 2>(a, 68, vec, blocks, s)));
  return launch_tri<T, 128, 4>(a, 96, vec, blocks, s);
}

template <typename T>
drpt_status launch_one(const LeafKnnArgs &a, unsigned blocks, cudaStream_t s) {
  const size_t smem = leaf_smem(a.k);
  DRPT_CUDA(cudaFuncSetAttribute(k_leaf_knn<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_leaf_knn<T><<<blocks, kThreads, smem, s>>>(a);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

}  // namespace

drpt_status launch_leaf_knn_exact(const LeafKnnArgs &a, cudaStream_t s) {
  if (a.k <= 0 || a.k > kMaxK) {
    set_error("leaf k-NN: k = %d outside [1, %d]", a.k, kMaxK);
    return DRPT_ERR_UNSUPPORTED;
  }
  const int64_t blocks = (int64_t)a.T * a.n_final;
  if (blocks <= 0) return DRPT_OK;
  if (blocks > 0x7fffffff) return DRPT_ERR_UNSUPPORTED;
  if (a.k <= 32) {
    DRPT_TRY(a.dtype == DRPT_DTYPE_U8 ? launch_tris<uint8_t>(a, (unsigned)blocks, s)
                                      : launch_tris<float>(a, (unsigned)blocks, s));
    return launch_leaf_tiles_exact(a, 128, s);
  }
  return a.dtype == DRPT_DTYPE_U8 ? launch_one<uint8_t>(a, (unsigned)blocks, s)
                                  : launch_one<float>(a, (unsigned)blocks, s);
}

int leaf_knn_exact_kernels(int k) { return k <= 32 ? 4 : 1; }

}  // namespace drpt
