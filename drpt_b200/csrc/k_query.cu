// Out-of-sample queries against the trees of a built index (no reference
// counterpart: the reference stores its splits, drpt_global.cpp:290 and
// drpt_local.cpp:142-155, but never reads them back).
//
//   Q1 k_descend  per (query, tree): walk the heap from the root with the
//                 query's projected values and the stored node medians,
//                 `value <= median` going left as in the build
//                 (drpt_global.cpp:308); ends at a global leaf
//   Q2            exact FP32 distances (sequential fused multiply-adds over
//                 the dimensions, square root) of the members of each query's
//                 leaf in every tree, and the k best of them by (distance,
//                 id): k_query_few reads a leaf for each query, k_query_tile
//                 once for all queries that fall in it
//   Q3            the trees' lists merged (a point found in several trees
//                 counts once): by the query's last block of k_query_few, or
//                 the builds' cross-tree merge
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "sm100.cuh"
#include "warp_list.cuh"

namespace drpt {
namespace {

__global__ void k_descend(const float *__restrict__ Pq, int64_t nq, int T, int gd,
                          const float *__restrict__ medians, int32_t *__restrict__ leaf) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nq * T) return;
  const int64_t q = e / T;
  const int t = (int)(e - q * T);
  const int nleaf = 1 << (gd - 1);
  const float *med = medians + (int64_t)t * (nleaf - 1);
  int node = 0;  // heap index; children of h are 2h+1 (left), 2h+2 (right)
  for (int l = 0; l + 1 < gd; ++l) {
    const float v = Pq[((int64_t)t * (gd - 1) + l) * nq + q];
    node = 2 * node + 1 + ((v <= __ldg(med + node)) ? 0 : 1);
  }
  leaf[e] = node - (nleaf - 1);
}

template <typename T>
__device__ __forceinline__ float4 ld4(const T *p);
template <>
__device__ __forceinline__ float4 ld4<float>(const float *p) {
  return __ldg(reinterpret_cast<const float4 *>(p));
}
template <>
__device__ __forceinline__ float4 ld4<uint8_t>(const uint8_t *p) {
  const uchar4 v = __ldg(reinterpret_cast<const uchar4 *>(p));
  return make_float4(v.x, v.y, v.z, v.w);
}

// The leaf of a query in tree t, by one warp: lane l sums the query's value of
// level l (as k_project does: the column's nonzeros in order, each product and
// sum rounded), then the walk of k_descend, kWalk levels at a time: lanes load
// the medians of the whole subtree below the node, so that a round of loads
// serves kWalk steps.
struct QueryTrees {
  const int32_t *colptr, *row;  // the trees' columns, T * (gd - 1)
  const float *val, *medians;   // T x (2^(gd-1) - 1), heap order
  int gd;
};
__device__ __forceinline__ int warp_descend(const QueryTrees &q, int t, const float *qv,
                                            int lane) {
  constexpr int kWalk = 5;
  const int levels = q.gd - 1;
  const float *med = q.medians + (int64_t)t * ((1 << levels) - 1);
  float v = 0.0f;
  if (lane < levels) {
    const int e0 = __ldg(q.colptr + t * levels + lane), e1 = __ldg(q.colptr + t * levels + lane + 1);
#pragma unroll 4
    for (int e = e0; e < e1; ++e) v = __fadd_rn(v, __fmul_rn(qv[__ldg(q.row + e)], __ldg(q.val + e)));
  }
  int node = 0;  // heap index; children of h are 2h + 1 (left), 2h + 2 (right)
  for (int l0 = 0; l0 < levels; l0 += kWalk) {
    // lane i holds heap node i of the subtree below `node`: depth dl, and the
    // (i + 1 - 2^dl)-th of that level
    const int dl = 31 - __clz(lane + 1);
    const int h = ((node + 1) << dl) - 1 + (lane + 1 - (1 << dl));
    const float m = dl < kWalk && l0 + dl < levels ? __ldg(med + h) : 0.0f;
    int at = 0;
    for (int i = 0; i < kWalk && l0 + i < levels; ++i) {
      const float x = __shfl_sync(kFull, v, l0 + i), mi = __shfl_sync(kFull, m, at);
      const int right = x <= mi ? 0 : 1;
      at = 2 * at + 1 + right;
      node = 2 * node + 1 + right;
    }
  }
  return node - ((1 << levels) - 1);
}

// L <- the 32 smallest of L and a list of k entries (sorted over the lanes,
// lanes from k on ignored) whose members may lie in L already; a member carries
// the same distance in both, so it is skipped.  `tmp`: 64 words of the warp.
__device__ __forceinline__ void warp_join(float &ld, int32_t &li, float d, int32_t id, int k,
                                          int lane, float *tmp) {
  bool fresh = lane < k && id >= 0;
  for (int j = 0; j < k; ++j) fresh &= __shfl_sync(kFull, li, j) != id;
  const unsigned m = __ballot_sync(kFull, fresh);
  if (m == 0) return;
  // the fresh entries side by side, still sorted
  int32_t *ti = reinterpret_cast<int32_t *>(tmp + 32);
  tmp[lane] = __int_as_float(0x7f800000);
  ti[lane] = -1;
  __syncwarp();
  const int at = __popc(m & ((1u << lane) - 1u));
  if (fresh) {
    tmp[at] = d;
    ti[at] = id;
  }
  __syncwarp();
  warp_merge32(ld, li, tmp[lane], ti[lane], lane);
  __syncwarp();  // tmp is reused
}

// Q2a, few queries: block (e, s) takes share s of the S shares of the members
// of query e / T's leaf in tree e % T; warps take 32 members at a time, a lane
// each.  Latency bounds it (one query: a few thousand members), so the members
// spread over T * S blocks of eight warps and a lane keeps kBurst 16-byte
// pieces of its row in flight; a whole leaf per query on one warp took 911 us
// for one query of 6 trees with 1,024-point leaves.  With `trees` the block
// also finds its leaf itself, and with `tickets` (one per query) the query's last
// block merges its lists into the result: one launch where four took 26 us of the
// GPU.  A block lifts its query's ticket to `turn` (the call's, in the upper 32
// bits) before it joins its warps' lists, which hides it (at the block's start it
// took 0.3 to 1 us), and then counts itself in the lower bits, by the same thread:
// nothing that an earlier call left there is counted.
constexpr int kFewWarps = 8;
template <typename T>
__global__ void __launch_bounds__(32 * kFewWarps) k_query_few(
    const T *__restrict__ X, int d, int64_t n, const T *__restrict__ Qx, int T_, int S,
    const int32_t *__restrict__ order, const int32_t *__restrict__ goff, int nleaf,
    const int32_t *__restrict__ leaf, QueryTrees trees, int k, int32_t *ci, float *cd,
    unsigned long long *tickets, unsigned long long turn, int32_t *__restrict__ oi,
    float *__restrict__ od) {
  constexpr int kBurst = 8;
  extern __shared__ __align__(16) float qv[];  // the query's d values
  __shared__ float sd[kFewWarps][32];
  __shared__ int32_t si[kFewWarps][32];
  __shared__ int leaf_sh;
  __shared__ float tmp[kFewWarps][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t e = blockIdx.x / S;
  const int s = (int)(blockIdx.x - e * S);
  const int64_t q = e / T_;
  const int t = (int)(e - q * T_);
  for (int c = threadIdx.x; c < d; c += blockDim.x) qv[c] = (float)Qx[q * d + c];
  int lf;
  if (trees.medians) {
    __syncthreads();
    if (warp == 0) {
      const int l = warp_descend(trees, t, qv, lane);
      if (lane == 0) leaf_sh = l;
    }
    __syncthreads();
    lf = leaf_sh;
  } else {
    lf = __ldg(leaf + e);
    __syncthreads();
  }
  const int32_t *go = goff + (int64_t)t * (nleaf + 1);
  const int32_t lo0 = __ldg(go + lf), m = __ldg(go + lf + 1) - lo0;
  const int32_t per = ((m + S - 1) / S + 31) & ~31;
  const int32_t lo = lo0 + min(s * per, m), hi = lo0 + min((s + 1) * per, m);
  const int32_t *ord = order + (int64_t)t * n;
  const float inf = __int_as_float(0x7f800000);
  float ld = inf;  // the list: lane j holds the j-th best
  int32_t li = -1;
  for (int32_t base = lo + 32 * warp; base < hi; base += 32 * kFewWarps) {
    const int32_t pos = base + lane;
    const int32_t p = pos < hi ? __ldg(ord + pos) : -1;
    const T *row = X + (int64_t)max(p, 0) * d;
    float acc = 0.0f;
    for (int c0 = 0; c0 < d; c0 += 4 * kBurst) {  // d % 4 == 0
      float4 x[kBurst];
#pragma unroll
      for (int i = 0; i < kBurst; ++i)
        if (c0 + 4 * i < d) x[i] = ld4<T>(row + c0 + 4 * i);
#pragma unroll
      for (int i = 0; i < kBurst; ++i)
        if (c0 + 4 * i < d) {
          const float4 y = *reinterpret_cast<const float4 *>(qv + c0 + 4 * i);
          float df = x[i].x - y.x;
          acc = fmaf(df, df, acc);
          df = x[i].y - y.y;
          acc = fmaf(df, df, acc);
          df = x[i].z - y.z;
          acc = fmaf(df, df, acc);
          df = x[i].w - y.w;
          acc = fmaf(df, df, acc);
        }
    }
    warp_take(ld, li, sqrtf(acc), p, k, lane);
  }
  if (tickets && threadIdx.x == 0) atomicMax(tickets + q, turn);
  sd[warp][lane] = ld;
  si[warp][lane] = li;
  __syncthreads();
  if (warp == 0) {
    for (int w = 1; w < kFewWarps; ++w) warp_merge32(ld, li, sd[w][lane], si[w][lane], lane);
    if (lane < k) {
      ci[(int64_t)blockIdx.x * k + lane] = li;
      cd[(int64_t)blockIdx.x * k + lane] = ld;
    }
    if (tickets) {
      __threadfence();
      __syncwarp();
      if (lane == 0) leaf_sh = atomicAdd(tickets + q, 1ull) == turn + (unsigned)(T_ * S) - 1u;
      __syncwarp();
      __threadfence();
    }
  }
  if (!tickets) return;
  __syncthreads();
  if (!leaf_sh) return;  // block-uniform
  // the query's last block: warps take its T * S lists in turn, warp 0 joins
  // the warps' lists
  ld = inf;
  li = -1;
  const int lists = T_ * S;
  for (int l0 = warp; l0 < lists; l0 += 4 * kFewWarps) {
    float d4[4];
    int32_t i4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int l = l0 + i * kFewWarps;
      const bool in = l < lists && lane < k;
      d4[i] = in ? __ldcg(cd + (q * lists + l) * k + lane) : inf;
      i4[i] = in ? __ldcg(ci + (q * lists + l) * k + lane) : -1;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) warp_join(ld, li, d4[i], i4[i], k, lane, tmp[warp]);
  }
  sd[warp][lane] = ld;
  si[warp][lane] = li;
  __syncthreads();
  if (warp != 0) return;
  for (int w = 1; w < min(kFewWarps, lists); ++w)
    warp_join(ld, li, sd[w][lane], si[w][lane], k, lane, tmp[0]);
  if (lane < k) {
    oi[q * k + lane] = li;
    od[q * k + lane] = li >= 0 ? ld : inf;
  }
}

// Many queries: the (query, tree) pairs grouped by leaf, so that a leaf's
// rows are staged once for up to QT queries.
//   k_query_count  pairs per (tree, leaf) and each pair's place among them
//   k_query_plan   leaf offsets in the grouped list, items of <= QT queries
//   k_query_fill   the grouped list
__global__ void k_query_count(const int32_t *__restrict__ leaf, int64_t nq, int T_, int nleaf,
                              int32_t *__restrict__ cnt, int32_t *__restrict__ rank) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nq * T_) return;
  rank[e] = atomicAdd(cnt + (int64_t)(e % T_) * nleaf + leaf[e], 1);
}

__global__ void __launch_bounds__(1024) k_query_plan(const int32_t *__restrict__ cnt, int B,
                                                     int qt, int32_t *__restrict__ off,
                                                     int4 *__restrict__ items,
                                                     int32_t *__restrict__ n_items) {
  __shared__ int tot[2][32];
  const int per = (B + 1023) / 1024;
  const int b0 = threadIdx.x * per, b1 = min(b0 + per, B);
  int c = 0, it = 0;
  for (int b = b0; b < b1; ++b) {
    c += cnt[b];
    it += (cnt[b] + qt - 1) / qt;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int xc = c, xi = it;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int yc = __shfl_up_sync(kFull, xc, o), yi = __shfl_up_sync(kFull, xi, o);
    if (lane >= o) {
      xc += yc;
      xi += yi;
    }
  }
  if (lane == 31) {
    tot[0][w] = xc;
    tot[1][w] = xi;
  }
  __syncthreads();
  if (w < 2) {
    int v = tot[w][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, v, o);
      if (lane >= o) v += y;
    }
    tot[w][lane] = v;
  }
  __syncthreads();
  int oc = xc - c + (w > 0 ? tot[0][w - 1] : 0), oi = xi - it + (w > 0 ? tot[1][w - 1] : 0);
  for (int b = b0; b < b1; ++b) {
    off[b] = oc;
    for (int q = 0; q < cnt[b]; q += qt) items[oi++] = make_int4(b, oc + q, min(qt, cnt[b] - q), 0);
    oc += cnt[b];
  }
  if (threadIdx.x == 1023) *n_items = oi;
}

__global__ void k_query_fill(const int32_t *__restrict__ leaf, const int32_t *__restrict__ rank,
                             const int32_t *__restrict__ off, int64_t nq, int T_, int nleaf,
                             int32_t *__restrict__ list) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nq * T_) return;
  list[off[(int64_t)(e % T_) * nleaf + leaf[e]] + rank[e]] = (int32_t)(e / T_);
}

// Q2b: one item (<= QT queries of one leaf) against every kMT-member tile of
// the leaf.  Members and queries are staged in kKc-dimension chunks, dimension
// major, through two shared buffers (the next chunk is in registers while the
// current one is used); thread (ty, tx) owns queries QT/16 ty + i and members
// 4 tx + j, 64 + 4 tx + j; a packed multiply-add takes two members at once,
// each pair's sum running over the dimensions in order as in k_query_few.
// Then the selection: warp w keeps the lists of queries w QT/8 .. in its
// lanes.  FP32 issue bounds it: two operations per dimension and pair.  50,000
// queries of 262,144 x 128 (6 trees, leaves of 1,024): 38.8 ms with a warp per
// query reading its leaves, 5.3 ms with QT = 64, 10 ms with QT = 16, which
// serves leaves with fewer queries (kQueryWide), where 64 would mostly compute
// padding (4,096 queries: 1.2 against 1.5 ms).
constexpr int kMT = 128, kKc = 32, kQThreads = 256;
constexpr int kSPitch = kMT + 4;
template <int QT>
constexpr size_t query_smem() {
  return sizeof(float) * (2 * kKc * kMT + 2 * kKc * QT + QT * kSPitch) +
         sizeof(int32_t) * (kMT + QT);
}

template <typename T, int QT>
__global__ void __launch_bounds__(kQThreads, 2) k_query_tile(
    const T *__restrict__ X, int d, int64_t n, const T *__restrict__ Qx, int T_,
    const int32_t *__restrict__ order, const int32_t *__restrict__ goff, int nleaf,
    const int4 *__restrict__ items, const int32_t *__restrict__ n_items,
    const int32_t *__restrict__ list, int k, int32_t *__restrict__ ci, float *__restrict__ cd) {
  constexpr int QPT = QT / 16;   // queries per thread
  constexpr int QPW = QT / 8;    // queries per warp in the selection
  constexpr int QG = QT * kKc / 4 / kQThreads > 0 ? QT * kKc / 4 / kQThreads : 1;  // query quads
  extern __shared__ __align__(16) float sm[];
  float *Ms = sm;                               // [2][kKc][kMT]
  float *Qs = Ms + 2 * kKc * kMT;               // [2][kKc][QT]
  float *St = Qs + 2 * kKc * QT;                // [QT][kSPitch]
  int32_t *cid = reinterpret_cast<int32_t *>(St + QT * kSPitch);  // kMT
  int32_t *qid = cid + kMT;                     // QT
  if ((int)blockIdx.x >= *n_items) return;
  const int4 item = items[blockIdx.x];
  const int t = item.x / nleaf, lf = item.x - t * nleaf, nqi = item.z;
  const int32_t *go = goff + (int64_t)t * (nleaf + 1);
  const int32_t lo = __ldg(go + lf), m = __ldg(go + lf + 1) - lo;
  const int32_t *ord = order + (int64_t)t * n + lo;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int warp = tid >> 5, lane = tid & 31;
  if (tid < QT) qid[tid] = tid < nqi ? __ldg(list + item.y + tid) : -1;
  __syncthreads();
  // staging: member sr, 16 dimensions from sk; query quads (row, 4 dimensions)
  const int sr = tid & (kMT - 1), sk = (tid >> 7) * 16;
  float4 pm[4], pq[QG];
  auto member = [&](int m0) { return m0 + sr < m ? __ldg(ord + m0 + sr) : -1; };
  auto fetch = [&](int32_t row, int k0) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = k0 + sk + 4 * i;
      pm[i] = row >= 0 && c < d ? ld4<T>(X + (int64_t)row * d + c) : z;
    }
#pragma unroll
    for (int i = 0; i < QG; ++i) {
      const int g = tid + i * kQThreads, r = g % QT, c = k0 + 4 * (g / QT);
      pq[i] = z;
      if (g < QT * (kKc / 4) && qid[r] >= 0 && c < d) pq[i] = ld4<T>(Qx + (int64_t)qid[r] * d + c);
    }
  };
  auto store = [&](int b) {
    float *M = Ms + b * kKc * kMT;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      M[(sk + 4 * i) * kMT + sr] = pm[i].x;
      M[(sk + 4 * i + 1) * kMT + sr] = pm[i].y;
      M[(sk + 4 * i + 2) * kMT + sr] = pm[i].z;
      M[(sk + 4 * i + 3) * kMT + sr] = pm[i].w;
    }
#pragma unroll
    for (int i = 0; i < QG; ++i) {
      const int g = tid + i * kQThreads, r = g % QT, c = 4 * (g / QT);
      if (g < QT * (kKc / 4)) {
        float *Q = Qs + (b * kKc + c) * QT + r;
        Q[0] = pq[i].x;
        Q[QT] = pq[i].y;
        Q[2 * QT] = pq[i].z;
        Q[3 * QT] = pq[i].w;
      }
    }
  };
  const float inf = __int_as_float(0x7f800000);
  float ld[QPW];
  int32_t li[QPW];
#pragma unroll
  for (int i = 0; i < QPW; ++i) {
    ld[i] = inf;
    li[i] = -1;
  }
  int32_t row = member(0);
  fetch(row, 0);
  for (int m0 = 0; m0 < m; m0 += kMT) {
    const int32_t next = member(m0 + kMT);
    float2 acc[QPT][4];
#pragma unroll
    for (int i = 0; i < QPT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    store(0);
    __syncthreads();  // chunk 0 stored; the previous tile's selection is done
    if (tid < kMT) cid[tid] = row;
    int cur = 0;
    for (int k0 = 0; k0 < d; k0 += kKc, cur ^= 1) {
      const bool more = k0 + kKc < d;
      if (more) fetch(row, k0 + kKc);
      else if (m0 + kMT < m) fetch(next, 0);
      const float *M = Ms + cur * kKc * kMT;
      const float *Q = Qs + cur * kKc * QT + QPT * ty;
      if (2 * QPT * warp < nqi)  // a warp of the item's queries (else all padding)
#pragma unroll 8
      for (int kk = 0; kk < kKc; ++kk) {
        const float4 a = *reinterpret_cast<const float4 *>(M + kk * kMT + 4 * tx);
        const float4 b = *reinterpret_cast<const float4 *>(M + kk * kMT + 64 + 4 * tx);
        const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float y[QPT];
        if constexpr (QPT == 4) {
          const float4 q = *reinterpret_cast<const float4 *>(Q + kk * QT);
          y[0] = q.x; y[1] = q.y; y[2] = q.z; y[3] = q.w;
        } else {
#pragma unroll
          for (int i = 0; i < QPT; ++i) y[i] = Q[kk * QT + i];
        }
#pragma unroll
        for (int i = 0; i < QPT; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 df = make_float2(x[2 * j] - y[i], x[2 * j + 1] - y[i]);
            acc[i][j] = sm100::fma2(df, df, acc[i][j]);
          }
      }
      // the other buffer was last read before the barrier that ended the
      // previous chunk
      if (more) {
        store(cur ^ 1);
        __syncthreads();
      }
    }
#pragma unroll
    for (int i = 0; i < QPT; ++i) {
      float *s = St + (QPT * ty + i) * kSPitch;
      *reinterpret_cast<float4 *>(s + 4 * tx) =
          make_float4(sqrtf(acc[i][0].x), sqrtf(acc[i][0].y), sqrtf(acc[i][1].x),
                      sqrtf(acc[i][1].y));
      *reinterpret_cast<float4 *>(s + 64 + 4 * tx) =
          make_float4(sqrtf(acc[i][2].x), sqrtf(acc[i][2].y), sqrtf(acc[i][3].x),
                      sqrtf(acc[i][3].y));
    }
    __syncthreads();  // scores and ids stored; every chunk read
#pragma unroll
    for (int i = 0; i < QPW; ++i) {
      const int q = warp * QPW + i;
      if (q < nqi) {  // warp-uniform
#pragma unroll
        for (int h = 0; h < kMT / 32; ++h)
          warp_take(ld[i], li[i], St[q * kSPitch + 32 * h + lane], cid[32 * h + lane], k, lane);
      }
    }
    row = next;
  }
#pragma unroll
  for (int i = 0; i < QPW; ++i) {
    const int q = warp * QPW + i;
    if (q < nqi && lane < k) {
      const int64_t o = ((int64_t)qid[q] * T_ + t) * k + lane;
      ci[o] = li[i];
      cd[o] = ld[i];
    }
  }
}

template <typename T, int QT>
drpt_status query_tile(const QueryArgs &a, unsigned max_items, cudaStream_t s) {
  constexpr size_t smem = query_smem<QT>();
  DRPT_CUDA(cudaFuncSetAttribute(k_query_tile<T, QT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_query_tile<T, QT><<<max_items, kQThreads, smem, s>>>(
      (const T *)a.X, a.d, a.n, (const T *)a.Q, a.T, a.order, a.goff, a.nleaf, a.items, a.n_items,
      a.list, a.k, a.ci, a.cd);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

// Queries per item of the grouped form; 0: the few-queries form.  The grouped
// form stages a leaf once for the queries that fall in it (nq / nleaf on
// average), the other one reads it for each query.  262,144 x 128, 256 leaves
// a tree: 512 queries (2 a leaf) take 0.46 ms with a leaf read per query and
// 0.75 grouped, 1,024 queries 0.84 and 0.86, 2,048 queries 1.6 and 0.88; with
// 64 instead of 16 an item 4,096 queries (16 a leaf) 1.5 against 1.2 ms, 8,192
// queries 1.6 against 2.0.
constexpr int kQueryWide = 24, kQueryGroup = 4;
int query_group(int64_t nq, int nleaf) {
  const int64_t per = nq / nleaf;
  return per >= kQueryWide ? 64 : (per >= kQueryGroup ? 16 : 0);
}

// Shares that the few-queries form cuts a leaf into: until the pairs fill the
// SMs, but no share below the block's 256 members.  More than one share only
// below kQueryTickets pairs (so queries): lists of shares are joined by the last
// block.
int64_t most_shares() { return std::min<int64_t>(8 * device_sm_count(), kQueryTickets); }
int64_t leaf_shares(int max_leaf) { return ceil_div(std::max(max_leaf, 1), 32 * kFewWarps); }
int query_shares(int64_t pairs, int max_leaf) {
  return (int)std::max<int64_t>(
      1, std::min(leaf_shares(max_leaf), most_shares() / std::max<int64_t>(pairs, 1)));
}

}  // namespace

drpt_status launch_descend(const float *Pq, int64_t nq, int T, int gd, const float *medians,
                           int32_t *leaf, cudaStream_t s) {
  if (nq <= 0) return DRPT_OK;
  k_descend<<<(unsigned)ceil_div(nq * T, 256), 256, 0, s>>>(Pq, nq, T, gd, medians, leaf);
  DRPT_LAUNCH_CHECK();
  return DRPT_OK;
}

// `aligned`: the query rows can be read in 16-byte (u8: 4-byte) pieces, as the
// grouped form does.  `random_only`: no tree splits on learned values.
constexpr int kQueryWalk = 32;
QueryPlan query_plan(int64_t nq, int T, int nleaf, int max_leaf, int k, bool aligned,
                     bool random_only) {
  QueryPlan p{};
  p.qt = aligned ? query_group(nq, nleaf) : 0;
  const int64_t pairs = nq * T;
  if (p.qt == 0) {
    p.shares = query_shares(pairs, max_leaf);
    p.lists = pairs * p.shares;
    // the block's own walk costs each of them about 4 us, two launches 10
    p.descend = random_only && nq <= kQueryWalk;
    p.join = nq <= kQueryTickets;
  } else {
    p.shares = 1;
    p.lists = pairs;
    p.buckets = (int64_t)T * nleaf;
    p.items = ceil_div(pairs, p.qt) + std::min<int64_t>(p.buckets, pairs);
  }
  p.entries = p.lists * k;
  return p;
}

QueryRoom query_room(int64_t cap, int T, int nleaf, int max_leaf, int k) {
  const int64_t pairs = cap * T;
  QueryRoom r{};
  // a list a pair, or the shares of few pairs
  r.entries = std::max(pairs, std::min(pairs * leaf_shares(max_leaf), most_shares())) * k;
  if (query_group(cap, nleaf) > 0) {  // (else no fewer queries are grouped)
    r.buckets = (int64_t)T * nleaf;
    r.items = ceil_div(pairs, 16) + std::min(r.buckets, pairs);
  }
  return r;
}

drpt_status launch_query(const QueryArgs &a, const QueryPlan &p, cudaStream_t s) {
  if (a.nq <= 0) return DRPT_OK;
  if (a.k <= 0 || a.k > 32 || a.d % 4 != 0 || a.d > 1024) {
    set_error("queries: k in [1, 32] and d %% 4 == 0, d <= 1024 (got k %d, d %d)", a.k, a.d);
    return DRPT_ERR_UNSUPPORTED;
  }
  const bool u8 = a.dtype == DRPT_DTYPE_U8;
  if (p.qt == 0) {
    if (p.lists > 0x7fffffff) {
      set_error("queries: %lld (query, tree) pairs in one launch", (long long)p.lists);
      return DRPT_ERR_UNSUPPORTED;
    }
    QueryTrees trees{};
    if (p.descend) trees = QueryTrees{a.csc.colptr, a.csc.row, a.csc.val, a.medians, a.gd};
    auto few = [&](auto *X, auto *Q) {
      using E = std::remove_const_t<std::remove_pointer_t<decltype(X)>>;
      k_query_few<E><<<(unsigned)p.lists, 32 * kFewWarps, a.d * sizeof(float), s>>>(
          X, a.d, a.n, Q, a.T, p.shares, a.order, a.goff, a.nleaf, a.leaf, trees, a.k, a.ci, a.cd,
          p.join ? a.tickets : nullptr, (unsigned long long)a.turn << 32, a.oi, a.od);
    };
    if (u8) few((const uint8_t *)a.X, (const uint8_t *)a.Q);
    else few((const float *)a.X, (const float *)a.Q);
    DRPT_LAUNCH_CHECK();
    if (p.join) return DRPT_OK;
  } else {
    const int64_t pairs = a.nq * a.T;
    const unsigned grid = (unsigned)ceil_div(pairs, 256);
    DRPT_CUDA(cudaMemsetAsync(a.cnt, 0, (size_t)p.buckets * 4, s));
    k_query_count<<<grid, 256, 0, s>>>(a.leaf, a.nq, a.T, a.nleaf, a.cnt, a.rank);
    k_query_plan<<<1, 1024, 0, s>>>(a.cnt, (int)p.buckets, p.qt, a.off, a.items, a.n_items);
    k_query_fill<<<grid, 256, 0, s>>>(a.leaf, a.rank, a.off, a.nq, a.T, a.nleaf, a.list);
    DRPT_LAUNCH_CHECK();
    const unsigned items = (unsigned)p.items;
    if (p.qt == 64)
      DRPT_TRY((u8 ? query_tile<uint8_t, 64>(a, items, s) : query_tile<float, 64>(a, items, s)));
    else
      DRPT_TRY((u8 ? query_tile<uint8_t, 16>(a, items, s) : query_tile<float, 16>(a, items, s)));
  }
  return launch_merge(a.ci, a.cd, a.nq, a.T, a.k, a.k, a.oi, a.od, s);
}

}  // namespace drpt
