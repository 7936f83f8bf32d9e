// Host-side, libstdc++-defined parts of the DRPT path (see host_algo.h).
#include "host_algo.h"

#include <algorithm>
#include <numeric>
#include <random>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace drpt {

namespace {

// std::mt19937's sequence (M. Matsumoto and T. Nishimura, "Mersenne Twister",
// 1998) made 624 outputs at a time, so that draws above a bound can be passed
// over many at once; a uniform random bit generator for libstdc++'s
// distributions.
class Mt19937 {
 public:
  using result_type = std::mt19937::result_type;
  static constexpr result_type min() { return std::mt19937::min(); }
  static constexpr result_type max() { return std::mt19937::max(); }
  Mt19937(uint32_t seed, uint32_t bound) : bound_(bound) {
    x_[0] = seed;
    for (uint32_t i = 1; i < kN; ++i) x_[i] = 1812433253u * (x_[i - 1] ^ (x_[i - 1] >> 30)) + i;
  }
  result_type operator()() {
    if (at_ == kN) refill();
    return out_[at_++];
  }
  // Skips draws above the bound, at most `most` of them; the number skipped.
  int64_t skip_above(int64_t most) {
    int64_t skipped = 0;
    while (skipped < most) {
      if (at_ == kN) refill();
      // the first marked draw from at_ on
      int w = at_ >> 6;
      uint64_t m = low_[w] >> (at_ & 63) << (at_ & 63);
      while (m == 0 && w < kN / 64) m = low_[++w];
      const int hit = m ? 64 * w + __builtin_ctzll(m) : kN;
      const int stop = (int)std::min<int64_t>(hit, at_ + (most - skipped));
      skipped += stop - at_;
      at_ = stop;
      if (stop < kN) break;
    }
    return skipped;
  }

 private:
  static constexpr int kN = 624, kM = 397;
  static uint32_t twist(uint32_t hi, uint32_t lo) {
    const uint32_t y = (hi & 0x80000000u) | (lo & 0x7fffffffu);
    return (y >> 1) ^ ((0u - (lo & 1u)) & 0x9908b0dfu);
  }
  // x_[i] for i in [from, to), each from x_[i + shift] (in place: a step of
  // four reads nothing that it or a later one writes)
  void twist_range(int from, int to, int shift) {
    int i = from;
#if defined(__SSE2__)
    const __m128i hi = _mm_set1_epi32(INT32_MIN), lo = _mm_set1_epi32(0x7fffffff);
    const __m128i one = _mm_set1_epi32(1), mat = _mm_set1_epi32((int32_t)0x9908b0dfu);
    for (; i + 4 <= to; i += 4) {
      const __m128i a = load(x_ + i), b = load(x_ + i + 1), c = load(x_ + i + shift);
      const __m128i y = _mm_or_si128(_mm_and_si128(a, hi), _mm_and_si128(b, lo));
      const __m128i odd = _mm_cmpeq_epi32(_mm_and_si128(b, one), one);
      store(x_ + i, _mm_xor_si128(c, _mm_xor_si128(_mm_srli_epi32(y, 1), _mm_and_si128(odd, mat))));
    }
#endif
    for (; i < to; ++i) x_[i] = x_[i + shift] ^ twist(x_[i], x_[i + 1]);
  }
  void refill() {
    twist_range(0, kN - kM, kM);
    twist_range(kN - kM, kN - 1, kM - kN);
    x_[kN - 1] = x_[kM - 1] ^ twist(x_[kN - 1], x_[0]);
    at_ = 0;
#if defined(__SSE2__)
    // tempered, and the draws at or below the bound marked
    const __m128i flip = _mm_set1_epi32(INT32_MIN);  // unsigned order as signed
    const __m128i bound = _mm_xor_si128(_mm_set1_epi32((int32_t)bound_), flip);
    const __m128i m1 = _mm_set1_epi32((int32_t)0x9d2c5680u);
    const __m128i m2 = _mm_set1_epi32((int32_t)0xefc60000u);
    std::fill(low_, low_ + kN / 64 + 1, 0ull);
    for (int i = 0; i < kN; i += 4) {
      __m128i y = load(x_ + i);
      y = _mm_xor_si128(y, _mm_srli_epi32(y, 11));
      y = _mm_xor_si128(y, _mm_and_si128(_mm_slli_epi32(y, 7), m1));
      y = _mm_xor_si128(y, _mm_and_si128(_mm_slli_epi32(y, 15), m2));
      y = _mm_xor_si128(y, _mm_srli_epi32(y, 18));
      store(out_ + i, y);
      const int above =
          _mm_movemask_ps(_mm_castsi128_ps(_mm_cmpgt_epi32(_mm_xor_si128(y, flip), bound)));
      low_[i >> 6] |= (uint64_t)(above ^ 15) << (i & 63);
    }
#else
    std::fill(low_, low_ + kN / 64 + 1, 0ull);
    for (int i = 0; i < kN; ++i) {
      uint32_t y = x_[i];
      y ^= y >> 11;
      y ^= (y << 7) & 0x9d2c5680u;
      y ^= (y << 15) & 0xefc60000u;
      out_[i] = y ^ (y >> 18);
      low_[i >> 6] |= (uint64_t)(out_[i] <= bound_) << (i & 63);
    }
#endif
  }
#if defined(__SSE2__)
  static __m128i load(const uint32_t *p) {
    return _mm_loadu_si128(reinterpret_cast<const __m128i *>(p));
  }
  static void store(uint32_t *p, __m128i v) { _mm_storeu_si128(reinterpret_cast<__m128i *>(p), v); }
#endif
  uint32_t x_[kN], out_[kN], bound_;
  uint64_t low_[kN / 64 + 1];  // bit i: draw i lies at or below the bound
  int at_ = kN;
};

// A generator that returns one given draw, and counts how often it is asked.
struct OneDraw {
  using result_type = std::mt19937::result_type;
  static constexpr result_type min() { return std::mt19937::min(); }
  static constexpr result_type max() { return std::mt19937::max(); }
  result_type operator()() {
    ++asked;
    return draw;
  }
  uint32_t draw;
  int asked = 0;
};

}  // namespace

// Row-major over d rows and L columns; one uniform draw per entry, and a
// normal draw only for the entries the uniform draw keeps.  The uniform value
// grows with its draw, so the entries it drops are those whose draw lies above
// a bound, found by bisection with libstdc++'s own distribution; they are most
// of the draws, and only looked through.
void host_projection_nonzeros(uint32_t seed, int d, int L, float density,
                              std::vector<Nonzero> *out) {
  out->clear();
  std::uniform_real_distribution<float> keep(0, 1);
  std::normal_distribution<float> gauss(0, 1);
  auto keeps = [&](uint32_t draw) {
    OneDraw g{draw};
    return !(keep(g) > density);
  };
  OneDraw probe{0u};
  keep(probe);
  const int64_t total = (int64_t)d * L;
  if (probe.asked != 1) {  // another standard library: entry by entry
    std::mt19937 gen(seed);
    for (int64_t e = 0; e < total; ++e) {
      const float u = keep(gen);
      const float v = (u > density) ? 0.0f : gauss(gen);
      if (v != 0.0f) out->push_back({(int32_t)(e / L), (int32_t)(e % L), v});
    }
    return;
  }
  if (!keeps(0u)) return;
  uint32_t lo = 0u, hi = 0xffffffffu;  // the largest kept draw lies in [lo, hi]
  while (lo < hi) {
    const uint32_t mid = lo + (uint32_t)(((uint64_t)hi - lo + 1) / 2);
    if (keeps(mid)) lo = mid;
    else hi = mid - 1;
  }
  Mt19937 gen(seed, lo);
  out->reserve((size_t)((double)total * std::min(1.0, 1.1 * ((double)lo + 1.0) / 4294967296.0)) + 16);
  int64_t row = 0, col = 0;
  for (int64_t e = 0; e < total; ++e, ++col) {
    const int64_t s = gen.skip_above(total - e);
    e += s;
    if (e >= total) break;
    col += s;
    if (col >= 8 * (int64_t)L) {
      row += col / L;
      col %= L;
    }
    for (; col >= L; col -= L) ++row;
    gen();  // the kept entry's uniform draw
    const float v = gauss(gen);
    if (v != 0.0f) out->push_back({(int32_t)row, (int32_t)col, v});
  }
}

void host_projection_matrix(uint32_t seed, int d, int L, float density, float *B) {
  std::vector<Nonzero> nz;
  host_projection_nonzeros(seed, d, L, density, &nz);
  std::fill(B, B + (int64_t)d * L, 0.0f);
  for (const Nonzero &z : nz) B[(int64_t)z.row * L + z.col] = z.val;
}

bool host_local_matrix_is_zero(uint32_t seed, int d, int L) {
  std::mt19937 gen(seed);
  std::uniform_real_distribution<float> keep(0, 1);
  std::normal_distribution<float> gauss(0, 1);
  for (int64_t e = 0; e < (int64_t)d * L; ++e) {
    const float u = keep(gen);
    if (!(u > 0.0f)) {
      if (gauss(gen) != 0.0f) return false;
    }
  }
  return true;
}

namespace {

void split_range(std::vector<int32_t>::iterator b, std::vector<int32_t>::iterator e, int depth,
                 int ld) {
  if (depth == ld) return;
  const int64_t size = e - b;
  // All local keys are zero, so the reference's `<` comparator is false for
  // every pair; nth_element's permutation then depends on the size only.
  std::nth_element(b, b + size / 2, e, [](int32_t, int32_t) { return false; });
  const auto mid = e - size / 2;  // left half keeps ceil(size / 2)
  split_range(b, mid, depth + 1, ld);
  split_range(mid, e, depth + 1, ld);
}

void sizes_rec(int64_t n, int level, int ld, std::vector<int32_t> &out) {
  if (level == ld) {
    out.push_back((int32_t)n);
    return;
  }
  sizes_rec(n - n / 2, level + 1, ld, out);
  sizes_rec(n / 2, level + 1, ld, out);
}

}  // namespace

void host_local_permutation(int64_t n, int ld, std::vector<int32_t> &perm,
                            std::vector<int32_t> &first) {
  perm.resize(n);
  std::iota(perm.begin(), perm.end(), 0);
  split_range(perm.begin(), perm.end(), 0, ld);
  std::vector<int32_t> sizes;
  sizes.reserve((size_t)1 << ld);
  sizes_rec(n, 0, ld, sizes);
  first.assign(sizes.size() + 1, 0);
  for (size_t l = 0; l < sizes.size(); ++l) first[l + 1] = first[l] + sizes[l];
}

namespace {

// The reference's candidate record (drpt_global.hpp:17-20): the same field
// order, so that std::sort sees the same sequence of comparisons and moves.
struct PriorityMap {
  int leaf_index;
  float priority;
};

}  // namespace

bool host_locality_slots(int T, int nleaf, int64_t n, const int32_t *order, const int32_t *goff,
                         int32_t *slot_leaf) {
  // every point's leaf in every tree (index_to_tree_leaf_mapper,
  // drpt_global.cpp:314, 323)
  std::vector<int32_t> leaf_of((size_t)n * T, 0);
  for (int t = 0; t < T; ++t)
    for (int j = 0; j < nleaf; ++j)
      for (int32_t i = goff[(size_t)t * (nleaf + 1) + j]; i < goff[(size_t)t * (nleaf + 1) + j + 1];
           ++i)
        leaf_of[(size_t)order[(size_t)t * n + i] * T + t] = j;
  // sel[(tree * nleaf + leaf) * T + c]: the first leaf of tree c holding the
  // largest share (count / size * 100, in float) of the points of `leaf` of
  // `tree` (drpt_global.cpp:607-652)
  std::vector<int32_t> sel((size_t)T * nleaf * T);
  std::vector<float> cnt((size_t)T * nleaf);
  for (int tree = 0; tree < T; ++tree)
    for (int leaf = 0; leaf < nleaf; ++leaf) {
      std::fill(cnt.begin(), cnt.end(), 0.0f);
      const int32_t lo = goff[(size_t)tree * (nleaf + 1) + leaf];
      const int32_t hi = goff[(size_t)tree * (nleaf + 1) + leaf + 1];
      const int size = hi - lo;
      for (int32_t i = lo; i < hi; ++i) {
        const int32_t p = order[(size_t)tree * n + i];
        for (int j = 0; j < T; ++j) cnt[(size_t)j * nleaf + leaf_of[(size_t)p * T + j]] += 1.0f;
      }
      for (int c = 0; c < T; ++c) {
        const float *x = cnt.data() + (size_t)c * nleaf;
        int best = 0;
        float bv = (x[0] / size) * 100;
        for (int l = 1; l < nleaf; ++l) {  // std::max_element: the first largest
          const float v = (x[l] / size) * 100;
          if (bv < v) {
            bv = v;
            best = l;
          }
        }
        sel[((size_t)tree * nleaf + leaf) * T + c] = best;
      }
    }
  // At one rank every candidate list holds one leaf at priority 1 (its
  // frequency among the ranks, sortByFreq) and the others at 0
  // (drpt_global.cpp:667-688).
  auto candidates = [&](int tree, int leaf, int m, std::vector<PriorityMap> &v) {
    v.resize(nleaf);
    const int s = sel[((size_t)tree * nleaf + leaf) * T + m];
    for (int q = 0; q < nleaf; ++q) v[q] = PriorityMap{q, q == s ? 1.0f : 0.0f};
  };
  // slots in ascending order, trees in order: the leaf of tree m at slot k
  // follows the leaf chosen for slot k in tree m - 1 (select_next_candidate,
  // drpt_global.cpp:104-151, and the loop at :690-699)
  std::vector<uint8_t> taken((size_t)T * nleaf, 0);  // leaf of tree m used by a lower slot
  std::vector<int32_t> zero_sel((size_t)T * T, 0);   // leaves of tree cur choosing leaf 0 of m
  for (int cur = 0; cur < T; ++cur)
    for (int j = 0; j < nleaf; ++j)
      for (int m = 0; m < T; ++m)
        if (sel[((size_t)cur * nleaf + j) * T + m] == 0) ++zero_sel[(size_t)cur * T + m];
  std::vector<PriorityMap> vec;
  for (int k = 0; k < nleaf; ++k) {
    int prev = k;
    for (int m = 0; m < T; ++m) {
      const int cur = m == 0 ? 0 : m - 1;
      // the sorted list starts with its one priority-1 leaf: when that leaf
      // is free it is the choice and the order of the rest does not matter
      const int top = sel[((size_t)cur * nleaf + prev) * T + m];
      if (!taken[(size_t)m * nleaf + top]) {
        slot_leaf[(size_t)k * T + m] = top;
        taken[(size_t)m * nleaf + top] = 1;
        prev = top;
        continue;
      }
      candidates(cur, prev, m, vec);
      std::sort(vec.begin(), vec.end(), [](const PriorityMap &lhs, const PriorityMap &rhs) {
        if (lhs.priority > rhs.priority) return true;
        return false;
      });
      int chosen = -1;
      for (const PriorityMap &can : vec) {
        const int id = can.leaf_index;
        if (taken[(size_t)m * nleaf + id]) continue;
        // another leaf j != prev of tree cur whose candidate list starts with
        // a higher-priority entry for the same leaf: only entry 0 is looked
        // at, which is leaf 0 with priority 1 exactly when j chose leaf 0
        if (id == 0 && can.priority < 1.0f) {
          const int others = zero_sel[(size_t)cur * T + m] -
                             (sel[((size_t)cur * nleaf + prev) * T + m] == 0 ? 1 : 0);
          if (others > 0) continue;
        }
        chosen = id;
        break;
      }
      if (chosen < 0) return false;
      slot_leaf[(size_t)k * T + m] = chosen;
      taken[(size_t)m * nleaf + chosen] = 1;
      prev = chosen;
    }
  }
  return true;
}

}  // namespace drpt
