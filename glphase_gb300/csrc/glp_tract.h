// glp_tract.h -- the runs of agreeing common sites behind the kNN
// tract-length metric (insti -T: the number of common sites minus
// Haplotype::MaxTractLen, src/haplotype.cpp:62-90, over the common sites of
// KNN::CutDownHaps, src/kNN.cpp:216-257), one 64-site word at a time.
//
// Plain C++ or CUDA: knn_tract_dist_kernel (glp_knn.cuh) runs these on the
// device; the host build lets the same code be checked on the CPU.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define GLP_TRACT_FN __host__ __device__ __forceinline__
#else
#define GLP_TRACT_FN inline
#endif

namespace glp {

GLP_TRACT_FN uint32_t tract_popc(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__popcll(x);
#else
  return (uint32_t)__builtin_popcountll(x);
#endif
}

// Lowest and highest set bit of x != 0.
GLP_TRACT_FN int tract_lsb(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return __ffsll((long long)x) - 1;
#else
  return __builtin_ctzll(x);
#endif
}

GLP_TRACT_FN int tract_msb(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return 63 - __clzll((long long)x);
#else
  return 63 - __builtin_clzll(x);
#endif
}

GLP_TRACT_FN uint32_t tract_max(uint32_t a, uint32_t b) { return a > b ? a : b; }

// Runs of agreeing common sites in a stretch of words: len common sites, pre
// of them before the first disagreement, suf after the last, best the longest
// run; pre == len when the stretch has no disagreement.
struct Tract {
  uint32_t len, pre, suf, best;
};

// One word: x the disagreements at common sites, m the common sites.
GLP_TRACT_FN Tract tract_word(uint64_t x, uint64_t m) {
  Tract t;
  t.len = tract_popc(m);
  if (x == 0) {
    t.pre = t.suf = t.best = t.len;
    return t;
  }
  const int lo = tract_lsb(x), hi = tract_msb(x);
  if (m == ~0ull) {  // every site common: the longest run of agreements in log steps
    const uint64_t r1 = ~x, r2 = r1 & (r1 >> 1), r4 = r2 & (r2 >> 2), r8 = r4 & (r4 >> 4),
                   r16 = r8 & (r8 >> 8), r32 = r16 & (r16 >> 16);
    // cur: the starts of runs of at least n agreements; n grows greedily
    uint64_t cur = ~0ull;
    uint32_t n = 0;
    const uint64_t rs[6] = {r32, r16, r8, r4, r2, r1};
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 6; ++i) {
      const uint64_t cand = cur & (rs[i] >> n);
      if (cand) {
        n += 32u >> i;
        cur = cand;
      }
    }
    t.pre = (uint32_t)lo;
    t.suf = (uint32_t)(63 - hi);
    t.best = n;
    return t;
  }
  t.pre = tract_popc(m & ((1ull << lo) - 1ull));
  t.suf = hi == 63 ? 0u : tract_popc(m >> (hi + 1));
  uint32_t best = tract_max(t.pre, t.suf);
  int prev = lo;
  for (uint64_t y = x & (x - 1ull); y; y &= y - 1ull) {  // runs between disagreements
    const int q = tract_lsb(y);                          // prev < q <= 63
    const uint64_t between = ((1ull << q) - 1ull) & ~((2ull << prev) - 1ull);
    best = tract_max(best, tract_popc(m & between));
    prev = q;
  }
  t.best = best;
  return t;
}

// The stretch l followed by the stretch r.
GLP_TRACT_FN Tract tract_join(const Tract l, const Tract r) {
  Tract t;
  t.len = l.len + r.len;
  t.pre = l.pre == l.len ? l.len + r.pre : l.pre;
  t.suf = r.suf == r.len ? r.len + l.suf : r.suf;
  t.best = tract_max(tract_max(l.best, r.best), l.suf + r.pre);
  return t;
}

// The runs of a pair over the stretch so far: `best` the longest, `open` the one
// that reaches its end.  best starts at kRunFloor: a pair that still has it at the
// end has no longer run, and its longest is found by tract_join.  That takes as
// long as all the other words together and its lanes wait for one another, so the
// floor is one that pairs practically never keep (haplotypes that agree at half of
// 1,024 sites at random have no run of 8 in one pair of eight: with a floor of 7
// the distances of 24,000 of them took 77 ms, 47 with this one).
struct OpenRun {
  uint32_t open, best;
};
constexpr uint32_t kRunFloor = 1;
// From which tract_inside32_any and _long may be used.
constexpr uint32_t kRunMid = 3, kRunLong = 7;

// The stretch followed by one word (x the disagreements at common sites, m the
// common sites).
GLP_TRACT_FN void tract_extend(OpenRun &r, uint64_t x, uint64_t m) {
  const Tract t = tract_word(x, m);
  r.best = tract_max(tract_max(r.best, t.best), r.open + t.pre);
  r.open = x == 0 ? r.open + t.len : t.suf;
}

// The stretch followed by 32 sites that are all common, but for the runs inside
// them: the runs that touch their ends come from the counts of leading and
// trailing zeros.
GLP_TRACT_FN void tract_extend32(OpenRun &r, uint32_t x) {
#if defined(__CUDA_ARCH__)
  const uint32_t low = (uint32_t)__clz((int)__brev(x)), high = (uint32_t)__clz((int)x);
#else
  const uint32_t low = x ? (uint32_t)__builtin_ctz(x) : 32u,
                 high = x ? (uint32_t)__builtin_clz(x) : 32u;
#endif
  r.best = tract_max(r.best, r.open + low);
  r.open = high + (x == 0 ? r.open : 0u);
}

// The runs inside 32 sites that are all common, which matter only beyond `best`
// (at least kRunFloor): two shifted starts of runs of 2, 4, 8 or 16 tell whether
// there is a longer one, and `best` goes up while there is.
GLP_TRACT_FN void tract_inside32(uint32_t &best, uint32_t x) {
  const uint32_t r1 = ~x, r2 = r1 & (r1 >> 1), r4 = r2 & (r2 >> 2), r8 = r4 & (r4 >> 4),
                 r16 = r8 & (r8 >> 8);
  for (;;) {  // bit i of `from`: a run of n starts at i; none starts past 32 - n
    const uint32_t from = best < 3 ? r2 : best < 7 ? r4 : best < 15 ? r8 : r16,
                   by = best - (best < 3 ? 1u : best < 7 ? 3u : best < 15 ? 7u : 15u);
    if (!(from & (from >> (by < 31u ? by : 31u))))
      break;
    ++best;
  }
}

// The same for `best` of at least kRunMid.
GLP_TRACT_FN void tract_inside32_any(uint32_t &best, uint32_t x) {
  const uint32_t r1 = ~x, r2 = r1 & (r1 >> 1), r4 = r2 & (r2 >> 2), r8 = r4 & (r4 >> 4),
                 r16 = r8 & (r8 >> 8);
  for (;;) {
    const uint32_t from = best < 7 ? r4 : best < 15 ? r8 : r16,
                   by = best - (best < 7 ? 3u : best < 15 ? 7u : 15u);
    if (!(from & (from >> (by < 31u ? by : 31u))))
      break;
    ++best;
  }
}

// The same for `best` of at least kRunLong.
GLP_TRACT_FN void tract_inside32_long(uint32_t &best, uint32_t x) {
  const uint32_t r1 = ~x, r2 = r1 & (r1 >> 1), r4 = r2 & (r2 >> 2), r8 = r4 & (r4 >> 4),
                 r16 = r8 & (r8 >> 8);
  for (;;) {
    const uint32_t from = best < 15 ? r8 : r16, by = best - (best < 15 ? 7u : 15u);
    if (!(from & (from >> (by < 31u ? by : 31u))))
      break;
    ++best;
  }
}

}  // namespace glp
