// K2-K4 -- one level of every global tree: node statistics, 16-slot
// histogram median and stable partition (drpt_global.cpp:228-352 with
// MathOp::distributed_mean/_variance/_median, math_operations.cpp:121-383, at
// one rank).
//
// A node's points are a contiguous range of the tree's `ord` array in
// ascending point index (the root starts in index order and every partition
// is stable); `val` holds the matching split values.  The work of a level is
// cut into units of up to kUnit consecutive positions that never straddle a
// node, so large nodes near the root spread over the whole GPU and small
// nodes near the leaves cost one unit each:
//
//   plan      a block per tree: units per node, their prefix, unit -> (node,
//             start).  Its own launch at the first level, afterwards one
//             extra block of the previous level's scatter launch
//   stats     exact: one block per node runs the reference's sequential FP32
//             sums (a single dependent add chain: warp 0 adds the values in
//             list order from a shared-memory double buffer that the other
//             warps fill); fast: FP64 partial sums per unit; the block that
//             finishes a node adds them in unit order and forms the node's
//             16 histogram boundaries (exact float arithmetic)
//   hist      per unit, 16 integer counts; the block that finishes a node
//             adds them, selects and interpolates the median (in double, as
//             the reference)
//   count     per unit, values <= median; the block that finishes a node
//             forms the units' prefix and the child offsets
//   scatter   per unit: warp-ballot stable partition through shared memory,
//             coalesced writes of the point ids and of their next-level values
//
// Where nodes are small a node of one unit runs through all of it inside the
// first of these kernels (exact: the histogram one), its values in registers
// from the first step to the last.  A level takes four launches (exact: five)
// where a launch per step took eight, and one when no node can exceed a unit
// (n <= kUnit).  Builds: 2,003 x 96, 8 trees, 0.57 -> 0.52 ms; 64 datasets x 96
// in one batch 27.9 -> 26.6 ms (its single-block plan of 262,144 node slots
// took 95 us per level); three 131,071 x 128 builds in a stream 6.67 -> 6.37.
//
// Every operation that the reference performs in float or double rounds on
// its own here (__f*_rn / __d*_rn), so with exact = 1 the medians, and hence
// the trees, are bit-identical to the reference's.
#include "kernels.cuh"

namespace drpt {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kUnit = 4096;                  // positions per unit
constexpr int kPer = kUnit / kThreads;       // positions per thread in a unit
constexpr int kChainChunk = 2048;            // values per shared-memory buffer of the chain

// ------------------------------------------------------------------ helpers
// Histogram boundaries (math_operations.cpp:252-288, factor 1, 7 bins):
// slots 0..13 around the mean at multiples of sigma/30, sigma/6 and sigma/2;
// slots 14 and 15 stay 0.
__device__ void node_bounds(float mu, float sigma, float *D) {
  const float s1 = __double2float_rn(__ddiv_rn((double)sigma, 30.0));
  const float s2 = __double2float_rn(__ddiv_rn((double)sigma, 6.0));
  const float s3 = __double2float_rn(__ddiv_rn((double)sigma, 2.0));
#pragma unroll
  for (int j = 1; j <= 4; ++j) {
    const float r = __fmul_rn((float)j, s1);
    D[6 + j] = __fadd_rn(mu, r);
    D[7 - j] = __fsub_rn(mu, r);
  }
#pragma unroll
  for (int j = 1; j <= 2; ++j) {
    const float r = __fadd_rn(sigma, __fmul_rn((float)j, s2));
    D[10 + j] = __fadd_rn(mu, r);
    D[3 - j] = __fsub_rn(mu, r);
  }
  const float r3 = __fadd_rn(__fmul_rn(2.0f, sigma), __fmul_rn(1.0f, s3));
  D[13] = __fadd_rn(mu, r3);
  D[0] = __fsub_rn(mu, r3);
  D[14] = 0.0f;
  D[15] = 0.0f;
}

// Slot of x (math_operations.cpp:292-308): slot j in 1..15 when
// D[j-1] < x <= D[j]; slot 0 when no slot takes it.  D[0..13] never
// decrease (offsets from the mean in increasing order, rounded
// monotonically) and D[14] = D[15] = 0, so for x <= D[13] the slot is the
// number of D[0..12] below x (0 when x <= D[0], and for a NaN x); above
// D[13] only slot 14 can take x, when x <= 0.  That count is found by a
// branch-free binary search over D[0..12] (a lower bound in a non-decreasing
// array; D[13] >= x closes it): four compares instead of thirteen, the same
// slot for every x, NaNs included (every compare with a NaN is false).
__device__ __forceinline__ int bin_of(const float *D, float x) {
  if (x > D[13]) return x <= 0.0f ? 14 : 0;
  const bool c8 = D[7] < x;                                              // >= 8 below
  const bool c4 = (c8 ? D[11] : D[3]) < x;                               // + 4
  const bool c2 = (c8 ? (c4 ? D[13] : D[9]) : (c4 ? D[5] : D[1])) < x;  // + 2
  const int s = (c8 ? 8 : 0) + (c4 ? 4 : 0) + (c2 ? 2 : 0);
  const float t = c8 ? (c4 ? D[12] : (c2 ? D[10] : D[8]))
                     : (c4 ? (c2 ? D[6] : D[4]) : (c2 ? D[2] : D[0]));
  return s + (t < x ? 1 : 0);                                           // + 1
}

// Median selection and interpolation (math_operations.cpp:333-375): the
// first slot whose running count (a float) reaches int(50*n/100); the
// interpolation runs in double from float boundaries and is stored as float.
// Slot -1 (read when slot 0 is selected) is 0, the preceding node's D[15].
__device__ float node_median(const float *D, const unsigned *hist, int64_t n) {
  float cfreq = 0.0f;
  const float target = (float)((50 * n) / 100);
  int sel = kBins - 1;
  for (int k = 0; k < kBins; ++k) {
    cfreq = __double2float_rn(__dadd_rn((double)cfreq, (double)hist[k]));
    if (cfreq >= target) {
      sel = k;
      break;
    }
  }
  const double count = (double)hist[sel];
  const float lo = sel > 0 ? D[sel - 1] : 0.0f;
  const float width = __fsub_rn(D[sel], lo);
  const double frac =
      __ddiv_rn(__dsub_rn((double)(n / 2), __dsub_rn((double)cfreq, count)), count);
  return __double2float_rn(__dadd_rn((double)lo, __dmul_rn(frac, (double)width)));
}

struct NodeRange {
  int64_t lo, hi;
};

__device__ __forceinline__ NodeRange node_range(const TreeLevelArgs &a, int g) {
  const int nodes = 1 << a.level;
  const int t = g >> a.level, s = g & (nodes - 1);
  if (!a.off_in) return {0, a.n};
  const int32_t *o = a.off_in + (int64_t)t * (nodes + 1);
  return {o[s], o[s + 1]};
}

__device__ __forceinline__ const float *tree_vals(const TreeLevelArgs &a, int t) {
  // The first level (p_level0) reads its values straight from P (column
  // t*(gd-1)): the points are still in index order there.
  return a.level == a.p_level0 ? a.P + (int64_t)t * (a.gd - 1) * a.n
                               : a.val_in + (int64_t)t * a.n;
}

// ------------------------------------------------------------------ units
struct Unit {
  int g, nu;          // node of all trees, its units
  NodeRange r;
  int64_t lo;
  int len;
};

__device__ __forceinline__ int64_t ceil_units(int64_t len) { return ceil_div(len, kUnit); }

// Planned units of tree t, and its u-th.  With a.direct every node has one.
__device__ __forceinline__ int tree_units(const TreeLevelArgs &a, int t) {
  return a.direct ? 1 << a.level : a.n_units[t];
}
__device__ __forceinline__ Unit unit_of(const TreeLevelArgs &a, int t, int u) {
  Unit x;
  if (a.direct) {
    x.g = (t << a.level) + u;
    x.r = node_range(a, x.g);
    x.lo = x.r.lo;
  } else {
    const int64_t i = t * a.unit_stride + u;
    x.g = a.unit_node[i];
    x.r = node_range(a, x.g);
    x.lo = a.unit_lo[i];
  }
  x.nu = (int)ceil_units(x.r.hi - x.r.lo);
  x.len = (int)min64(kUnit, x.r.hi - x.lo);
  return x;
}
// First unit of node g (an index of the unit arrays).
__device__ __forceinline__ int64_t node_units(const TreeLevelArgs &a, int g) {
  return (int64_t)(g >> a.level) * a.unit_stride + a.node_ubase[g];
}

// Units of tree t's 2^level nodes from their starts `off`, and cleared
// tickets, by one block.
__device__ void plan_tree(const UnitPlan &p, const int32_t *off, int64_t n, int t, int level,
                          int64_t stride, unsigned *tickets) {
  constexpr int kRun = 4;  // consecutive nodes per thread and step
  __shared__ int warp_tot[32];
  const int nodes = 1 << level, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  int carry = 0;
  for (int s0 = 0; s0 < nodes; s0 += blockDim.x * kRun) {
    const int s1 = s0 + threadIdx.x * kRun;
    int32_t o[kRun + 1];
    int cnt = 0;
#pragma unroll
    for (int i = 0; i <= kRun; ++i) {
      const int s = min(s1 + i, nodes);
      o[i] = off ? off[s] : (s == 0 ? 0 : (int32_t)n);
    }
#pragma unroll
    for (int i = 0; i < kRun; ++i) cnt += (int)ceil_units(o[i + 1] - o[i]);
    int x = cnt;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const int y = __shfl_up_sync(kFull, x, k);
      if (lane >= k) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    int base = carry + x - cnt, all = 0;
    for (int k = 0; k < nw; ++k) {
      const int y = warp_tot[k];
      if (k < w) base += y;
      all += y;
    }
    carry += all;
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
      const int s = s1 + i;
      if (s >= nodes) break;
      const int g = (t << level) + s;
      p.node_ubase[g] = base;
      tickets[g] = 0u;
      const int nu = (int)ceil_units(o[i + 1] - o[i]);
      for (int c = 0; c < nu; ++c) {
        p.unit_node[t * stride + base + c] = g;
        p.unit_lo[t * stride + base + c] = (int32_t)(o[i] + (int64_t)c * kUnit);
      }
      base += nu;
    }
    __syncthreads();  // warp_tot is reused by the next step
  }
  if (threadIdx.x == 0) p.n_units[t] = carry;
}

__global__ void __launch_bounds__(1024) k_plan(TreeLevelArgs a) {
  const int t = blockIdx.x;
  const UnitPlan p{a.node_ubase, a.unit_node, a.unit_lo, a.n_units};
  plan_tree(p, a.off_in ? a.off_in + (int64_t)t * ((1 << a.level) + 1) : nullptr, a.n, t, a.level,
            a.unit_stride, a.tickets);
}

// Whether this unit is the last of the node's `nu` units to end step `step`
// (each unit takes a ticket per step): then every unit's results of the step
// are visible to this warp.  Called by the one warp that wrote the unit's
// results.
__device__ __forceinline__ bool last_of_node(const TreeLevelArgs &a, const Unit &x, int step) {
  __threadfence();
  __syncwarp();
  unsigned old = 0u;
  if ((threadIdx.x & 31) == 0) old = atomicAdd(a.tickets + x.g, 1u);
  if (__shfl_sync(kFull, old, 0) != (unsigned)(step + 1) * (unsigned)x.nu - 1u) return false;
  __threadfence();
  return true;
}

// Batches: root slot s0 of the first level owns the nodes s0 << depth ..
// below it; from depth stop[s0] on its nodes keep every point (the median is
// +inf, and the columns they would split on are all 0).
__device__ __forceinline__ bool stopped(const TreeLevelArgs &a, int g) {
  if (!a.stop) return false;
  const int depth = a.level - a.p_level0;
  return depth >= a.stop[(g & ((1 << a.level) - 1)) >> depth];
}

// The median of node g, kept (also in heap order) and returned.
__device__ __forceinline__ float keep_median(const TreeLevelArgs &a, int g, float med) {
  const int nodes = 1 << a.level, t = g >> a.level, s = g & (nodes - 1);
  if (stopped(a, g)) med = __int_as_float(0x7f800000);
  a.node_med[g] = med;
  if (a.medians) a.medians[(int64_t)t * ((1 << (a.gd - 1)) - 1) + (nodes - 1) + s] = med;
  return med;
}

// Child offsets of node g, whose left child gets `nleft` points.
__device__ __forceinline__ void keep_children(const TreeLevelArgs &a, int g, const NodeRange &r,
                                              int nleft) {
  const int nodes = 1 << a.level, t = g >> a.level, s = g & (nodes - 1);
  int32_t *oo = a.off_out + (int64_t)t * (2 * nodes + 1);
  oo[2 * s] = (int32_t)r.lo;
  oo[2 * s + 1] = (int32_t)(r.lo + nleft);
  if (s == nodes - 1) oo[2 * nodes] = (int32_t)r.hi;
}

// An empty node has no unit: its (NaN) median and child offsets.
__device__ void keep_empty(const TreeLevelArgs &a, int g, const NodeRange &r) {
  float D[kBins];
  unsigned h[kBins];
  const float nan = __int_as_float(0x7fffffff);
  node_bounds(nan, nan, D);
  for (int j = 0; j < kBins; ++j) h[j] = 0u;
  keep_median(a, g, node_median(D, h, 0));
  keep_children(a, g, r, 0);
}
__device__ __forceinline__ void keep_empty_nodes(const TreeLevelArgs &a, int t) {
  const int nodes = 1 << a.level;
  for (int s = threadIdx.x; s < nodes; s += blockDim.x) {
    const NodeRange r = node_range(a, (t << a.level) + s);
    if (r.lo == r.hi) keep_empty(a, (t << a.level) + s, r);
  }
}

// The unit's values, all loads of a thread in flight (position threadIdx.x +
// j * kThreads).
__device__ __forceinline__ void load_values(const TreeLevelArgs &a, int t, const Unit &x,
                                            float *xs) {
  const float *v = tree_vals(a, t) + x.lo;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int i = threadIdx.x + j * kThreads;
    xs[j] = i < x.len ? __ldg(v + i) : 0.0f;
  }
}

// ------------------------------------------------------------------ exact stats
// Sequential FP32 sum of v[0..n) (or of (v - mu)^2), warp 0 adding from a
// shared-memory double buffer that warps 1..7 fill.  All of warp 0 computes
// the same chain; every thread returns it after the final barrier.
template <bool kSq>
__device__ float block_chain(const float *__restrict__ v, int64_t n, float mu, float *buf,
                             float *result) {
  const int warp = threadIdx.x >> 5;
  const int64_t chunks = ceil_div(n, kChainChunk);
  float s = 0.0f;
  auto load = [&](int64_t c) {
    float *dst = buf + (c & 1) * kChainChunk;
    const int64_t base = c * kChainChunk;
    const int len = (int)min64(kChainChunk, n - base);
    for (int i = threadIdx.x - 32; i < len; i += kThreads - 32) {
      float x = __ldg(v + base + i);
      if (kSq) {
        const float df = __fsub_rn(x, mu);
        x = __fmul_rn(df, df);
      }
      dst[i] = x;
    }
  };
  if (warp != 0 && chunks > 0) load(0);
  for (int64_t c = 0; c < chunks; ++c) {
    __syncthreads();  // buffer c complete; buffer c+1 free
    if (warp != 0) {
      if (c + 1 < chunks) load(c + 1);
    } else {
      const float *src = buf + (c & 1) * kChainChunk;
      const int len = (int)min64(kChainChunk, n - c * kChainChunk);
      const int len4 = len & ~3;
      const float4 *src4 = reinterpret_cast<const float4 *>(src);
      auto add = [&](const float4 &q) {
        s = __fadd_rn(s, q.x);
        s = __fadd_rn(s, q.y);
        s = __fadd_rn(s, q.z);
        s = __fadd_rn(s, q.w);
      };
      int i = 0;
      if (len == kChainChunk) {
        // two register buffers of 32 values: one loads while the other's are
        // added, so that the chain waits for nothing but its own additions
        constexpr int kQ = 8, kGroups = kChainChunk / 4 / kQ;
        static_assert(kGroups % 2 == 0, "two buffers in turn");
        float4 q0[kQ], q1[kQ];
#pragma unroll
        for (int e = 0; e < kQ; ++e) q0[e] = src4[e];
#pragma unroll 1
        for (int g = 0; g < kGroups; g += 2) {
#pragma unroll
          for (int e = 0; e < kQ; ++e) q1[e] = src4[(g + 1) * kQ + e];
#pragma unroll
          for (int e = 0; e < kQ; ++e) add(q0[e]);
#pragma unroll
          for (int e = 0; e < kQ; ++e) q0[e] = src4[min(g + 2, kGroups - 1) * kQ + e];
#pragma unroll
          for (int e = 0; e < kQ; ++e) add(q1[e]);
        }
        i = len4 / 4;
      }
#pragma unroll 4
      for (; i < len4 / 4; ++i) add(src4[i]);
      for (int e = len4; e < len; ++e) s = __fadd_rn(s, src[e]);
    }
  }
  if (threadIdx.x == 0) *result = s;
  __syncthreads();
  return *result;
}

__global__ void __launch_bounds__(kThreads) k_stats_exact(TreeLevelArgs a) {
  __shared__ __align__(16) float buf[2 * kChainChunk];
  __shared__ float sh[2];
  const int g = blockIdx.x;
  const int t = g >> a.level;
  const NodeRange r = node_range(a, g);
  const int64_t cnt = r.hi - r.lo;
  const float *v = tree_vals(a, t) + r.lo;
  const float sum = block_chain<false>(v, cnt, 0.0f, buf, &sh[0]);     // :137-142
  const float mu = __fdiv_rn(sum, __int2float_rn((int)cnt));          // :164
  const float sq = block_chain<true>(v, cnt, mu, buf, &sh[1]);        // :186-192
  if (threadIdx.x == 0) {
    const float var = __fdiv_rn(sq, __int2float_rn((int)cnt - 1));    // :201
    float Dl[kBins];
    node_bounds(mu, __fsqrt_rn(var), Dl);
    float *D = a.node_D + (int64_t)g * kBins;
#pragma unroll
    for (int j = 0; j < kBins; ++j) D[j] = Dl[j];
  }
}

// ------------------------------------------------------------------ histogram
// Counts of the unit's values per slot, left in `tot` (shared, kBins) for the
// whole block.  Per thread, the 16 counts are 8-bit fields of two 64-bit
// registers (at most kPer = 16 values per thread), widened to 16-bit fields of
// four registers (a warp's sum is at most 512) and added over the warp with
// shuffles; no atomics.
__device__ __forceinline__ void block_hist(const float *xs, int len, const float *Ds,
                                           unsigned (*hist)[kBins], unsigned *tot) {
  float D[kBins];
#pragma unroll
  for (int j = 0; j < kBins; ++j) D[j] = Ds[j];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  static_assert(kPer < 256, "a thread's counts fit 8-bit fields");
  uint64_t c2[2] = {0ull, 0ull};
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (threadIdx.x + j * kThreads < len) {
      const int b = bin_of(D, xs[j]);
      const uint64_t inc = 1ull << (8 * (b & 7));
      c2[0] += b < 8 ? inc : 0ull;
      c2[1] += b < 8 ? 0ull : inc;
    }
  }
  // bins 4q .. 4q + 3 as 16-bit fields of c4[q]
  uint64_t c4[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t x = (uint32_t)(c2[q >> 1] >> (32 * (q & 1)));
    c4[q] = (uint64_t)(x & 0xffu) | ((uint64_t)((x >> 8) & 0xffu) << 16) |
            ((uint64_t)((x >> 16) & 0xffu) << 32) | ((uint64_t)(x >> 24) << 48);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c4[q] += __shfl_xor_sync(kFull, c4[q], o);
  const int q = lane >> 2;
  const uint64_t mine = q == 0 ? c4[0] : q == 1 ? c4[1] : q == 2 ? c4[2] : c4[3];
  if (lane < kBins) hist[w][lane] = (unsigned)((mine >> (16 * (lane & 3))) & 0xffffu);
  __syncthreads();
  if (threadIdx.x < kBins) {
    unsigned s = 0;
    for (int k = 0; k < kWarps; ++k) s += hist[k][threadIdx.x];
    tot[threadIdx.x] = s;
  }
  __syncthreads();
}

// ------------------------------------------------------------------ partition
// Warp-ballot stable partition of a unit through shared memory.  Position
// p = threadIdx.x + j * kThreads is chunk c = j * kWarps + warp of 32
// positions (so c-major order is position order); each warp's ballot of
// "value <= median" (goes left, drpt_global.cpp:308) gives the chunk's left
// count and, per lane, the left-goers before it in the chunk; one warp scans
// the kUnit / 32 chunk counts.  A left-goer lands at (left-goers before it), a
// right-goer at (left total + right-goers before it): left-goers in position
// order, then right-goers in position order.  All loads are coalesced; the
// point ids and their next-level values then leave in coalesced writes.
struct PartSmem {
  int32_t sid[kUnit];
  float sval[kUnit];
  int cbase[kUnit / 32];  // chunk left counts, then their exclusive prefix
  int ltot;
};

// `ids`: the unit's point ids in position order; the unit's left-goers go to
// lbase + .., its right-goers to rbase + .. (rbase < 0: behind the left-goers,
// a node of one unit).  Returns the left total; the caller's next use of `sm`
// needs a barrier first.
__device__ __forceinline__ int block_partition(const TreeLevelArgs &a, int t, const Unit &x,
                                               const float *xs, const int32_t *ids, float med,
                                               int64_t lbase, int64_t rbase, PartSmem &sm) {
  constexpr int kChunks = kUnit / 32;
  static_assert(kChunks == 4 * 32, "one warp scans the chunk counts, four per lane");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int len = x.len;
  unsigned bal[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int p = threadIdx.x + j * kThreads;
    bal[j] = __ballot_sync(kFull, p < len && xs[j] <= med);
    if (lane == 0) sm.cbase[j * kWarps + w] = __popc(bal[j]);
  }
  __syncthreads();
  if (w == 0) {
    int c4[4], sum = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      c4[e] = sm.cbase[4 * lane + e];
      sum += c4[e];
    }
    int y = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(kFull, y, o);
      if (lane >= o) y += z;
    }
    int run = y - sum;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      sm.cbase[4 * lane + e] = run;
      run += c4[e];
    }
    if (lane == 31) sm.ltot = y;
  }
  __syncthreads();
  const int ltot = sm.ltot;
  const bool want_val = a.val_out != nullptr;
  const float *pnext =
      want_val ? a.P + ((int64_t)t * (a.gd - 1) + a.level - a.p_level0 + 1) * a.n : nullptr;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int p = threadIdx.x + j * kThreads;
    if (p < len) {
      const int lbefore = sm.cbase[j * kWarps + w] + __popc(bal[j] & lt_mask);
      const int slot = ((bal[j] >> lane) & 1u) ? lbefore : ltot + (p - lbefore);
      sm.sid[slot] = ids[j];
      if (want_val) sm.sval[slot] = __ldg(pnext + ids[j]);
    }
  }
  __syncthreads();
  if (rbase < 0) rbase = lbase + ltot;
  int32_t *oout = a.ord_out + (int64_t)t * a.n;
  float *vout = want_val ? a.val_out + (int64_t)t * a.n : nullptr;
  for (int i = threadIdx.x; i < len; i += kThreads) {
    const int64_t dst = i < ltot ? lbase + i : rbase + (i - ltot);
    oout[dst] = sm.sid[i];
    if (want_val) vout[dst] = sm.sval[i];
  }
  return ltot;
}

__device__ __forceinline__ void load_ids(const TreeLevelArgs &a, int t, const Unit &x,
                                         int32_t *ids) {
  const int32_t *oin = a.ord_in ? a.ord_in + (int64_t)t * a.n + x.lo : nullptr;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int p = threadIdx.x + j * kThreads;
    ids[j] = p < x.len ? (oin ? __ldg(oin + p) : (int32_t)(x.lo + p)) : 0;
  }
}

// The rest of the level for a node of one unit, from its boundaries on.
__device__ __forceinline__ void finish_node(const TreeLevelArgs &a, int t, const Unit &x,
                                            const float *xs, const int32_t *ids, const float *Ds,
                                            unsigned (*hist)[kBins], unsigned *tot, float *med_sh,
                                            PartSmem &sm) {
  block_hist(xs, x.len, Ds, hist, tot);
  if (threadIdx.x == 0) {
    float D[kBins];
    unsigned h[kBins];
#pragma unroll
    for (int j = 0; j < kBins; ++j) {
      D[j] = Ds[j];
      h[j] = tot[j];
    }
    *med_sh = keep_median(a, x.g, node_median(D, h, x.len));
  }
  __syncthreads();
  const int ltot = block_partition(a, t, x, xs, ids, *med_sh, x.r.lo, -1, sm);
  if (threadIdx.x == 0) keep_children(a, x.g, x.r, ltot);
  __syncthreads();  // the shared arrays are reused by the next unit
}

// ------------------------------------------------------------------ fast stats
__device__ __forceinline__ void fast_bounds(double s1, double s2, int64_t cnt, float *D) {
  const double dn = (double)cnt;
  double var = (s2 - s1 * (s1 / dn)) / (dn - 1.0);
  if (var < 0.0) var = 0.0;  // rounding can push a zero variance below 0 (NaN stays NaN)
  node_bounds((float)(s1 / dn), __fsqrt_rn((float)var), D);
}

// FUSE: finishes the nodes of one unit (and then the later kernels skip them),
// chosen where the nodes average below two units: the registers of the later
// steps cost the sums of large nodes their occupancy.
template <bool FUSE>
__global__ void __launch_bounds__(kThreads, FUSE ? 4 : 6) k_stats(TreeLevelArgs a) {
  __shared__ double sh[2 * kWarps];
  const int t = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.y == 0) keep_empty_nodes(a, t);
  const int units = tree_units(a, t);
  for (int u = blockIdx.y; u < units; u += gridDim.y) {
    const Unit x = unit_of(a, t, u);
    if (x.len <= 0) continue;  // an empty node of the direct form
    if (stopped(a, x.g)) {
      // every point stays where it is, in the left child
      const int32_t *oin = a.ord_in ? a.ord_in + (int64_t)t * a.n + x.lo : nullptr;
      int32_t *oout = a.ord_out + (int64_t)t * a.n + x.lo;
      for (int i = threadIdx.x; i < x.len; i += kThreads)
        oout[i] = oin ? __ldg(oin + i) : (int32_t)(x.lo + i);
      if (threadIdx.x == 0 && x.lo == x.r.lo) {
        keep_median(a, x.g, 0.0f);
        keep_children(a, x.g, x.r, (int)(x.r.hi - x.r.lo));
      }
      continue;
    }
    const bool whole = FUSE && x.nu == 1;
    float xs[kPer];
    load_values(a, t, x, xs);
    double s1 = 0.0, s2 = 0.0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (threadIdx.x + j * kThreads < x.len) {
        const double v = (double)xs[j];
        s1 += v;
        s2 += v * v;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_down_sync(kFull, s1, o);
      s2 += __shfl_down_sync(kFull, s2, o);
    }
    if (lane == 0) {
      sh[2 * w] = s1;
      sh[2 * w + 1] = s2;
    }
    __syncthreads();
    double t1 = 0.0, t2 = 0.0;  // thread 0: the unit's sums
    if (threadIdx.x == 0) {
      for (int i = 0; i < kWarps; ++i) {
        t1 += sh[2 * i];
        t2 += sh[2 * i + 1];
      }
    }
    if constexpr (FUSE) {
      __shared__ unsigned hist[kWarps][kBins];
      __shared__ unsigned tot[kBins];
      __shared__ float Ds[kBins];
      __shared__ float med_sh;
      __shared__ PartSmem sm;
      if (whole) {
        if (threadIdx.x == 0) {
          float D[kBins];
          fast_bounds(t1, t2, x.len, D);
#pragma unroll
          for (int j = 0; j < kBins; ++j) Ds[j] = D[j];
        }
        int32_t ids[kPer];
        load_ids(a, t, x, ids);
        __syncthreads();  // Ds
        finish_node(a, t, x, xs, ids, Ds, hist, tot, &med_sh, sm);
        continue;
      }
    }
    if (w == 0) {
      if (lane == 0) {
        const int64_t i = t * a.unit_stride + u;
        a.unit_s[2 * i] = t1;
        a.unit_s[2 * i + 1] = t2;
      }
      if (last_of_node(a, x, 0)) {
        // lanes take the node's units in turn, the lane partials are then
        // added in a fixed tree order
        const int64_t u0 = node_units(a, x.g);
        double b1 = 0.0, b2 = 0.0;
        for (int64_t i = u0 + lane; i < u0 + x.nu; i += 32) {
          b1 += __ldcg(a.unit_s + 2 * i);
          b2 += __ldcg(a.unit_s + 2 * i + 1);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          b1 += __shfl_xor_sync(kFull, b1, o);
          b2 += __shfl_xor_sync(kFull, b2, o);
        }
        if (lane == 0) {
          float D[kBins];
          fast_bounds(b1, b2, x.r.hi - x.r.lo, D);
#pragma unroll
          for (int j = 0; j < kBins; ++j) a.node_D[(int64_t)x.g * kBins + j] = D[j];
        }
      }
    }
    __syncthreads();  // sh is reused by the next unit
  }
}

// Nodes that k_stats has finished.
__device__ __forceinline__ bool done_in_stats(const TreeLevelArgs &a, const Unit &x) {
  return (a.fuse && x.nu == 1) || stopped(a, x.g);
}

// ------------------------------------------------------------------ histogram and median
// EXACT: the first kernel of the units (k_stats_exact has left the boundaries),
// so it finishes the nodes of one unit.
template <bool EXACT>
__global__ void __launch_bounds__(kThreads) k_hist(TreeLevelArgs a) {
  __shared__ unsigned hist[kWarps][kBins];
  __shared__ unsigned tot[kBins];
  __shared__ float Ds[kBins];
  const int t = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (EXACT && blockIdx.y == 0) keep_empty_nodes(a, t);
  const int units = tree_units(a, t);
  for (int u = blockIdx.y; u < units; u += gridDim.y) {
    const Unit x = unit_of(a, t, u);
    if (x.len <= 0 || (!EXACT && done_in_stats(a, x))) continue;
    float xs[kPer];
    load_values(a, t, x, xs);
    if (threadIdx.x < kBins) Ds[threadIdx.x] = a.node_D[(int64_t)x.g * kBins + threadIdx.x];
    __syncthreads();
    if constexpr (EXACT) {
      if (x.nu == 1) {
        __shared__ float med_sh;
        __shared__ PartSmem sm;
        int32_t ids[kPer];
        load_ids(a, t, x, ids);
        finish_node(a, t, x, xs, ids, Ds, hist, tot, &med_sh, sm);
        continue;
      }
    }
    block_hist(xs, x.len, Ds, hist, tot);
    if (w == 0 && lane < kBins) a.unit_hist[(t * a.unit_stride + u) * kBins + lane] = tot[lane];
    if (w == 0 && last_of_node(a, x, EXACT ? 0 : 1)) {
      // lanes add the counts of the node's units in turn (integer counts, so
      // the order is immaterial), lane 0 selects the median
      const int64_t u0 = node_units(a, x.g);
      unsigned h[kBins];
#pragma unroll
      for (int j = 0; j < kBins; ++j) h[j] = 0u;
      for (int64_t i = u0 + lane; i < u0 + x.nu; i += 32)
#pragma unroll
        for (int j = 0; j < kBins; ++j) h[j] += __ldcg(a.unit_hist + i * kBins + j);
#pragma unroll
      for (int j = 0; j < kBins; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) h[j] += __shfl_xor_sync(kFull, h[j], o);
      if (lane == 0) {
        float D[kBins];
#pragma unroll
        for (int j = 0; j < kBins; ++j) D[j] = Ds[j];
        keep_median(a, x.g, node_median(D, h, x.r.hi - x.r.lo));
      }
    }
    __syncthreads();  // Ds is reused by the next unit
  }
}

// ------------------------------------------------------------------ count and child offsets
__global__ void __launch_bounds__(kThreads) k_count(TreeLevelArgs a) {
  __shared__ int sh[kWarps];
  const int t = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int units = tree_units(a, t);
  for (int u = blockIdx.y; u < units; u += gridDim.y) {
    const Unit x = unit_of(a, t, u);
    if (a.exact ? x.nu == 1 : done_in_stats(a, x)) continue;
    float xs[kPer];
    load_values(a, t, x, xs);
    const float med = a.node_med[x.g];
    int c = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j)  // value <= median goes left (drpt_global.cpp:308)
      c += (threadIdx.x + j * kThreads < x.len && xs[j] <= med) ? 1 : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(kFull, c, o);
    if (lane == 0) sh[w] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int k = 0; k < kWarps; ++k) tot += sh[k];
      a.unit_left[t * a.unit_stride + u] = tot;
    }
    if (w == 0 && last_of_node(a, x, a.exact ? 1 : 2)) {
      // exclusive prefix of the units' left counts in unit order, 32 units
      // per step with a running carry
      const int64_t u0 = node_units(a, x.g);
      int carry = 0;
      for (int i0 = 0; i0 < x.nu; i0 += 32) {
        const int i = i0 + lane;
        const int v = i < x.nu ? __ldcg(a.unit_left + u0 + i) : 0;
        int y = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int z = __shfl_up_sync(kFull, y, o);
          if (lane >= o) y += z;
        }
        if (i < x.nu) a.unit_lbase[u0 + i] = carry + y - v;
        carry += __shfl_sync(kFull, y, 31);
      }
      if (lane == 0) {
        a.node_nleft[x.g] = carry;
        keep_children(a, x.g, x.r, carry);
      }
    }
    __syncthreads();  // sh is reused by the next unit
  }
}

// ------------------------------------------------------------------ scatter
// The last block of every tree's row of blocks plans the next level's units
// instead (a.next).
__global__ void __launch_bounds__(kThreads) k_scatter(TreeLevelArgs a) {
  __shared__ PartSmem sm;
  const int t = blockIdx.x;
  if (a.next.n_units && blockIdx.y == gridDim.y - 1) {
    plan_tree(a.next, a.off_out + (int64_t)t * ((2 << a.level) + 1), a.n, t, a.level + 1,
              a.next_stride, a.tickets);
    return;
  }
  const int units = tree_units(a, t), step = gridDim.y - (a.next.n_units ? 1 : 0);
  for (int u = blockIdx.y; u < units; u += step) {
    const Unit x = unit_of(a, t, u);
    if (a.exact ? x.nu == 1 : done_in_stats(a, x)) continue;
    float xs[kPer];
    int32_t ids[kPer];
    load_values(a, t, x, xs);
    load_ids(a, t, x, ids);
    // left-goers -> [node lo + unit lbase, ...), right-goers -> [node lo + nleft + rbase, ...)
    const int64_t ul = a.unit_lbase[t * a.unit_stride + u];
    block_partition(a, t, x, xs, ids, a.node_med[x.g], x.r.lo + ul,
                    x.r.lo + a.node_nleft[x.g] + (x.lo - x.r.lo - ul), sm);
    __syncthreads();  // sm is reused by the next unit
  }
}

}  // namespace

drpt_status launch_tree_level(TreeLevelArgs a, bool first, bool last, cudaStream_t s, int *launches) {
  const int64_t G = (int64_t)a.T << a.level;
  a.unit_stride = tree_level_max_units(a.n, 1, a.level);
  if (G > (1 << 20) || a.unit_stride * a.T > 0x7fffffff) {
    set_error("too many tree nodes at level %d", a.level);
    return DRPT_ERR_UNSUPPORTED;
  }
  // every node one unit: no plan, and k_stats (exact: k_hist) does the rest
  a.direct = a.n <= kUnit ? 1 : 0;
  a.fuse = a.direct || (a.n >> a.level) < 2 * kUnit ? 1 : 0;
  const int64_t per_tree = a.direct ? (int64_t)1 << a.level : a.unit_stride;
  // unit kernels loop over the units actually planned
  const dim3 U((unsigned)a.T,
               (unsigned)min64(per_tree, ceil_div((int64_t)device_sm_count() * 16, a.T)));
  // the unit tables of odd levels lie behind those of even ones, so that the
  // scatter can plan the next level while it reads this one's
  const UnitPlan even{a.node_ubase, a.unit_node, a.unit_lo, a.n_units};
  const UnitPlan odd{a.node_ubase + a.max_nodes, a.unit_node + a.max_units,
                     a.unit_lo + a.max_units, a.n_units + a.T};
  const UnitPlan &mine = a.level & 1 ? odd : even;
  a.node_ubase = mine.node_ubase;
  a.unit_node = mine.unit_node;
  a.unit_lo = mine.unit_lo;
  a.n_units = mine.n_units;
  a.next = UnitPlan{};
  int k = 0;
  if (first && !a.direct) {
    k_plan<<<(unsigned)a.T, 1024, 0, s>>>(a);
    ++k;
  }
  if (a.exact) {
    k_stats_exact<<<(unsigned)G, kThreads, 0, s>>>(a);
    k_hist<true><<<U, kThreads, 0, s>>>(a);
    k += 2;
  } else {
    if (a.fuse) k_stats<true><<<U, kThreads, 0, s>>>(a);
    else k_stats<false><<<U, kThreads, 0, s>>>(a);
    ++k;
    if (!a.direct) {
      k_hist<false><<<U, kThreads, 0, s>>>(a);
      ++k;
    }
  }
  if (!a.direct) {
    k_count<<<U, kThreads, 0, s>>>(a);
    dim3 V = U;
    if (!last) {
      a.next = a.level & 1 ? even : odd;
      a.next_stride = tree_level_max_units(a.n, 1, a.level + 1);
      V.y += 1;
    }
    k_scatter<<<V, kThreads, 0, s>>>(a);
    k += 2;
  }
  DRPT_LAUNCH_CHECK();
  if (launches) *launches += k;
  return DRPT_OK;
}

int64_t tree_level_max_units(int64_t n, int T, int level) {
  return (int64_t)T * (ceil_div(n, kUnit) + ((int64_t)1 << level));
}

}  // namespace drpt
