// glp_knn.cuh -- kNN surrogate restriction on the device: the reference's
// KNN::ClusterHaps (src/kNN.cpp:123-206) with the Hamming metric
// (src/haplotype.cpp:35-60) or the tract-length metric (insti -T: the number
// of common sites minus Haplotype::MaxTractLen, src/haplotype.cpp:62-90,
// kNN.cpp:157-164) over the common sites of KNN::CutDownHaps
// (src/kNN.cpp:216-257).
//
// For each sample s of the H/2 samples: the ceil(K/2) haplotypes nearest to
// haplotype 2s, then the ceil(K/2) nearest to haplotype 2s+1 that are not
// already chosen, interleaved.  The sample's own haplotypes are excluded.
// Ties are ordered by haplotype index, a total order; the reference sorts
// with the unstable std::sort (kNN.cpp:172-173), so its tie order is
// implementation-defined.
//
// Distances, a chunk of samples at a time through global memory: Hamming as a
// matrix product (knn_gemm_kernel, glp_knn_gemm.cuh), or the tract length
// (knn_tract_dist_kernel: each word's runs of agreeing common sites --
// before its first disagreement, after its last, the longest between --
// joined in site order, glp_tract.h).  Selection (knn_select_kernel): one CTA
// per sample, its two rows of distances in registers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "glp_knn_plan.h"
#include "glp_tract.h"

namespace glp {

constexpr int kKnnThreads = 512;
constexpr uint32_t kKnnMaxHaps = 50000;
constexpr uint32_t kKnnMaxHalf = 1024;
constexpr uint16_t kKnnExcluded = 0xffffu;
constexpr uint32_t kKnnNoHap = 0xffffffffu;  // a list without distances behind it
constexpr int kGemmTimeout = 2;  // error flag bit: a wait of knn_gemm_kernel ran out

// The bits of 32 lanes transposed: lane l gets bit l of every lane's x (in some
// order, which a population count does not see).
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x, uint32_t lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int s = 16; s; s >>= 1, m ^= m << s) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? ((x & ~m) | ((y >> s) & m)) : ((x & m) | ((y << s) & ~m));
  }
  return x;
}

// Bit m of mask: site m's alt-allele frequency (or MAF) lies in [lb, ub].  One
// block per word: each warp takes 32 haplotypes at a time and counts the 64
// sites by transposing their bits.  Bound: the words' latency, a few loads a
// thread (20,000 haplotypes x 64 words: 1,757 us with one thread a site walking
// all haplotypes, 22 us this way).
constexpr int kCommonThreads = 1024;
__global__ void __launch_bounds__(kCommonThreads)
    common_sites_kernel(const uint64_t *__restrict__ haps, uint32_t H, uint32_t wn, uint32_t S,
                        double lb, double ub, int use_maf, uint64_t *__restrict__ mask) {
  __shared__ uint32_t cnt[64];
  const uint32_t w = blockIdx.x, lane = threadIdx.x & 31u;
  if (threadIdx.x < 64)
    cnt[threadIdx.x] = 0;
  __syncthreads();
  uint32_t lo = 0, hi = 0;  // of sites `lane` and 32 + lane
#pragma unroll 4
  for (uint32_t h0 = threadIdx.x - lane; h0 < H; h0 += kCommonThreads) {
    const uint32_t h = h0 + lane;
    const uint64_t x = h < H ? __ldg(haps + (size_t)h * wn + w) : 0ull;
    lo += __popc(warp_transpose((uint32_t)x, lane));
    hi += __popc(warp_transpose((uint32_t)(x >> 32), lane));
  }
  atomicAdd(&cnt[lane], lo);
  atomicAdd(&cnt[32 + lane], hi);
  __syncthreads();
  if (threadIdx.x < 64) {
    const uint32_t m = w * 64 + threadIdx.x;
    double af = (double)cnt[threadIdx.x] / H;
    if (use_maf)
      af = fabs(fabs(af - 0.5) - 0.5);
    const uint32_t bits = __ballot_sync(0xffffffffu, m < S && af >= lb && af <= ub);
    if (lane == 0)
      reinterpret_cast<uint32_t *>(mask + w)[threadIdx.x >> 5] = bits;
  }
}

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *red) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0)
    red[warp] = v;
  __syncthreads();
  uint32_t t = 0;
#pragma unroll
  for (int i = 0; i < kKnnThreads / 32; ++i)
    t += red[i];
  return t;
}

// Exclusive prefix over threads (thread order), block total in *total.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *red,
                                                    uint32_t *total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o)
      inc += n;
  }
  __syncthreads();
  if (lane == 31)
    red[warp] = inc;
  __syncthreads();
  uint32_t base = 0, all = 0;
#pragma unroll
  for (int i = 0; i < kKnnThreads / 32; ++i) {
    if ((uint32_t)i < warp)
      base += red[i];
    all += red[i];
  }
  *total = all;
  return base + inc - v;
}

// The selection.  A block takes one sample; each of its two rows of distances is
// read once, into registers (8 consecutive ones a vector).  A bound on the half-th smallest
// comes from the threads' minima -- at least `half` distances are at most the
// half-th smallest minimum -- by a binary search that costs one counting barrier a
// step; the entries up to the bound are collected and put in (distance, index)
// order by counting, for each, how many are smaller.  Where fewer threads than
// `half` hold a distance the bound is the half-th smallest itself, by a search that
// counts all of the registers' distances, or, up to kSelectAll haplotypes, all are
// collected (a table of 1,000 haplotypes x 1,000 sites, half = 200, takes 75 us with
// the search and 175 with all collected; 400, 100, 62 and 66; 300, 100, 60 and 59; 100,
// 25, 56 and 52).
// Rows that leave more than kSelectMost entries (many equal distances) take the
// general path: the exact threshold by a binary search over all distances, ties in
// index order by a block scan, a bitonic sort.
// Bound: instructions and the search's barriers (10,000 samples, 20,000
// haplotypes, half = 100: 0.40 ms; 2.29 ms with the general path for every row,
// one block an SM with its rows in shared memory).
constexpr uint32_t kSelectMost = 1024, kSelectAll = 320;

// The general path: the `half` smallest (d, index) of the entries of row d that
// are not kKnnExcluded and not in `taken` (may be null), written sorted to
// out[0 .. half); 0xffff, which no haplotype has, where the row holds fewer.
// keys: kKnnMaxHalf words.
__device__ __noinline__ void select_general(const uint16_t *__restrict__ d, uint32_t H,
                                            uint32_t half, uint32_t dmax, const uint32_t *taken,
                                            uint32_t *keys, uint32_t *red, uint32_t *out) {
  const uint32_t tid = threadIdx.x;
  auto at = [&](uint32_t h) -> uint32_t {
    return taken && ((taken[h >> 5] >> (h & 31u)) & 1u) ? (uint32_t)kKnnExcluded
                                                        : (uint32_t)__ldg(d + h);
  };
  // smallest t with #{d <= t} >= half
  uint32_t lo = 0, hi = dmax;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    uint32_t c = 0;
    for (uint32_t h = tid; h < H; h += kKnnThreads)
      c += at(h) <= mid ? 1u : 0u;  // mid < kKnnExcluded
    if (block_sum(c, red) >= half)
      hi = mid;
    else
      lo = mid + 1;
  }
  const uint32_t t = lo;
  const uint32_t chunk = (H + kKnnThreads - 1) / kKnnThreads;
  const uint32_t b0 = min(H, tid * chunk), b1 = min(H, b0 + chunk);
  uint32_t ties = 0, nless = 0;
  for (uint32_t h = b0; h < b1; ++h) {
    const uint32_t v = at(h);
    ties += v == t ? 1u : 0u;
    nless += v < t ? 1u : 0u;
  }
  uint32_t total, below;
  uint32_t rank = block_exclusive(ties, red, &total);
  uint32_t pos = block_exclusive(nless, red, &below);
  const uint32_t need = half - below;  // ties at t, taken in index order
  uint32_t n2 = 1;  // the next power of two
  while (n2 < half)
    n2 <<= 1;
  for (uint32_t i = tid; i < n2; i += kKnnThreads)
    keys[i] = 0xffffffffu;
  __syncthreads();
  // entries below the threshold first (positions [0, below)), then ties
  for (uint32_t h = b0; h < b1; ++h) {
    const uint32_t v = at(h);
    if (v < t) {
      keys[pos++] = (v << 16) | h;
    } else if (v == t) {
      if (rank < need)
        keys[below + rank] = (v << 16) | h;
      ++rank;
    }
  }
  __syncthreads();
  // bitonic sort of (distance, index)
  for (uint32_t k = 2; k <= n2; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = tid; i < n2; i += kKnnThreads) {
        const uint32_t l = i ^ j;
        if (l > i) {
          const uint32_t x = keys[i], y = keys[l];
          if ((x > y) == ((i & k) == 0)) {
            keys[i] = y;
            keys[l] = x;
          }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = tid; i < half; i += kKnnThreads)
    out[i] = keys[i] & 0xffffu;
  __syncthreads();
}

// The `half` nearest of row d into out, sorted; kV vectors of 8 distances a
// thread cover the row.
template <int kV>
__device__ __forceinline__ void select_nearest(const uint16_t *__restrict__ d, uint32_t H,
                                               uint32_t half, uint32_t dmax,
                                               const uint32_t *taken, uint32_t *keys,
                                               uint32_t *red, uint32_t *out, const int *error,
                                               int &flags) {
  const uint32_t tid = threadIdx.x;
  __shared__ uint32_t found, counts[3];
  uint4 v[kV];
#pragma unroll
  for (int i = 0; i < kV; ++i) {
    const uint32_t h = 8 * (i * kKnnThreads + tid);
    v[i] = h < H ? __ldg(reinterpret_cast<const uint4 *>(d + h))
                 : make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
    if (h < H && h + 8 > H) {  // H is even: whole pairs of entries past it
      if (h + 2 >= H)
        v[i].y = 0xffffffffu;
      if (h + 4 >= H)
        v[i].z = 0xffffffffu;
      v[i].w = 0xffffffffu;
    }
    const uint32_t gone = kV == 1 && taken && h < H ? (taken[h >> 5] >> (h & 31u)) & 255u : 0u;
    if (gone) {  // bits to halves of the words
      v[i].x |= (gone & 1u) * 0xffffu | (gone >> 1 & 1u) * 0xffff0000u;
      v[i].y |= (gone >> 2 & 1u) * 0xffffu | (gone >> 3 & 1u) * 0xffff0000u;
      v[i].z |= (gone >> 4 & 1u) * 0xffffu | (gone >> 5 & 1u) * 0xffff0000u;
      v[i].w |= (gone >> 6 & 1u) * 0xffffu | (gone >> 7 & 1u) * 0xffff0000u;
    }
  }
  if (error)  // beside the row's loads
    flags = *error;
  if (tid == 0)
    found = counts[0] = 0;
  // the least distance of each thread; the pitch's padding is excluded like an own
  // haplotype
  uint32_t least = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < kV; ++i) {
    least = __vminu2(least, __vminu2(__vminu2(v[i].x, v[i].y), __vminu2(v[i].z, v[i].w)));
  }
  least = min(least & 0xffffu, least >> 16);
  // smallest u with at least `want` threads' minima <= u, or distances where too few
  // threads hold one.  In wide rows the taken ones, at most `half`, are still there
  // (taking them out of the registers first cost the fourth block an SM).
  const int want = (int)(kV > 1 && taken ? 2 * half : half);
  uint32_t lo = 0, hi = dmax + 1;
  const bool bounded = __syncthreads_count(least <= dmax) >= want;
  while (bounded && lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__syncthreads_count(least <= mid) >= want)
      hi = mid;
    else
      lo = mid + 1;
  }
  if (!bounded)
    lo = hi = dmax;
  // wider rows give every thread a distance
  if (kV == 1 && !bounded && H > kSelectAll) {
    lo = 0;
    // a step's count is cleared one step ahead, when all have read its last value
    for (uint32_t now = 0; lo < hi;) {
      const uint32_t mid = (lo + hi) >> 1, mid2 = mid | mid << 16, next = now == 2 ? 0 : now + 1;
      uint32_t c = 0;
#pragma unroll
      for (int i = 0; i < kV; ++i)
        c += __vsetleu2(v[i].x, mid2) + __vsetleu2(v[i].y, mid2) + __vsetleu2(v[i].z, mid2) +
             __vsetleu2(v[i].w, mid2);
      c = __reduce_add_sync(0xffffffffu, (c & 0xffffu) + (c >> 16));
      if ((tid & 31u) == 0 && c)
        atomicAdd(&counts[now], c);
      if (tid == 0)
        counts[next] = 0;
      __syncthreads();
      if (counts[now] >= half)
        hi = mid;
      else
        lo = mid + 1;
      now = next;
    }
  }
  const uint32_t u = lo;
  if (least <= u) {
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      const uint32_t x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t dist = (x[j >> 1] >> (16 * (j & 1))) & 0xffffu;
        if (dist <= u) {
          const uint32_t h = 8 * (i * kKnnThreads + tid) + j;
          if (kV == 1 || !(taken && ((taken[h >> 5] >> (h & 31u)) & 1u))) {
            const uint32_t n = atomicAdd(&found, 1u);
            if (n < kSelectMost)
              keys[n] = (dist << 16) | h;
          }
        }
      }
    }
  }
  __syncthreads();
  const uint32_t n = found;
  if (n > kSelectMost || n < half) {  // the same for every thread
    __syncthreads();
    select_general(d, H, half, dmax, taken, keys, red, out);
    return;
  }
  for (uint32_t i = tid; i < ((n + 3) & ~3u); i += kKnnThreads)
    if (i >= n)
      keys[i] = 0xffffffffu;
  __syncthreads();
  for (uint32_t i = tid; i < n; i += kKnnThreads) {
    const uint32_t key = keys[i];
    uint32_t rank = 0;
    for (uint32_t j = 0; j < n; j += 4) {
      const uint4 o = *reinterpret_cast<const uint4 *>(keys + j);
      rank += (o.x < key) + (o.y < key) + (o.z < key) + (o.w < key);
    }
    if (rank < half)
      out[rank] = key & 0xffffu;
  }
  __syncthreads();
}

// Tiled tract-length distances (-T) of the query haplotypes [q0, q0 + nq) (2 s
// and 2 s + 1 for the samples s of a chunk) against every haplotype: the words
// 8 at a time, word-major in shared memory; each pair carries its open and its
// longest run of agreeing common sites through the words (words whose sites are
// all common, nearly all of them, as two 32-bit halves); the distance is the common
// sites minus the longest run.  A CTA takes 32 queries x 64 haplotypes, each
// thread 2 x 4 pairs.  kSym: the queries are the whole panel; tiles below the
// diagonal are not computed, their distances are written transposed.
// Words go in two passes (see below), or, the first `exact` chunks of 8, in one with
// each word's longest run found on its own, whose cost is the same for all
// haplotypes (tract_exact_chunks).
// Bound: the ALU instructions of a pair's word (89 % of that pipe).  4,990
// haplotypes x 1,024 sites, a table: 2.15 ms with all tiles in one pass, 0.77 with
// the tiles of one half in two; of haplotypes that agree at half of the sites at random
// (no long runs: `best` rises for longer, and every lane waits) 2.15 and 1.02.  The
// test inside has three forms; with a fourth for `best` from 3 to 14 0.773 and 1.10
// (more code to fetch), with two 0.792 and 1.20.  20,000 x 4,096 119 -> 34 ms.
constexpr uint32_t kTractQ = 32, kTractH = 64, kDistW = 8, kDistThreads = 256;
template <bool kSym>
__global__ void __launch_bounds__(kDistThreads)
    knn_tract_dist_kernel(const uint64_t *__restrict__ haps, uint32_t H, uint32_t wn,
                          const uint64_t *__restrict__ mask, uint32_t q0, uint32_t nq,
                          uint32_t pitch, uint32_t exact, uint16_t *__restrict__ dist) {
  const uint32_t hb = blockIdx.x * kTractH, qb = blockIdx.y * kTractQ;
  if (kSym && hb + kTractH <= qb)
    return;
  __shared__ uint64_t sq[kDistW][kTractQ];
  __shared__ uint64_t sh[kDistW][kTractH];
  __shared__ uint64_t smask[kDistW];
  __shared__ uint16_t st[kSym ? kTractH : 1][kTractQ + 2];  // the tile transposed
  const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
  const uint32_t chunks = (wn + kDistW - 1) / kDistW;
  const bool all_exact = chunks <= exact;
  uint32_t common = 0;
  int form = 0;  // of the test inside: 0 tract_inside32, 1 _any, 2 _long
  OpenRun run[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      run[i][j] = OpenRun{0, all_exact ? 0u : kRunFloor};
  // twice over the words: the runs that cross 32-site boundaries (and all of the
  // runs of exact words, and of words with sites that are not common), which leave
  // `best` near the longest; then the runs inside, which seldom exceed it
#pragma unroll 1
  for (uint32_t chunk = 0; chunk < 2 * chunks - exact; ++chunk) {
    const bool inside = chunk >= chunks;
    const uint32_t w0 = (inside ? chunk - chunks + exact : chunk) * kDistW;
    for (uint32_t i = tid; i < kTractQ * kDistW; i += kDistThreads) {
      const uint32_t r = i / kDistW, k = i % kDistW, w = w0 + k;
      sq[k][r] = (qb + r < nq && w < wn) ? __ldg(haps + (size_t)(q0 + qb + r) * wn + w) : 0ull;
    }
    for (uint32_t i = tid; i < kTractH * kDistW; i += kDistThreads) {
      const uint32_t r = i / kDistW, k = i % kDistW, w = w0 + k;
      sh[k][r] = (hb + r < H && w < wn) ? __ldg(haps + (size_t)(hb + r) * wn + w) : 0ull;
    }
    if (tid < kDistW)
      smask[tid] = w0 + tid < wn ? __ldg(mask + w0 + tid) : 0ull;
    __syncthreads();
    const uint32_t kn = min(kDistW, wn - w0);
    for (uint32_t k = 0; k < kn; ++k) {
      const uint64_t m = smask[k];
      uint64_t qv[2], hv[4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        qv[i] = sq[k][2 * ty + i];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        hv[j] = sh[k][tx + 16 * j];
      if (inside) {
        if (m == ~0ull) {
          // the form of the test that all of the warp's pairs may use
          if (form != 2) {
            uint32_t least = run[0][0].best;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                least = min(least, run[i][j].best);
            form = __all_sync(0xffffffffu, least >= kRunLong)  ? 2
                   : __all_sync(0xffffffffu, least >= kRunMid) ? 1
                                                               : 0;
          }
          auto inside_word = [&](auto test) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                test(run[i][j].best, (uint32_t)(qv[i] ^ hv[j]));
                test(run[i][j].best, (uint32_t)((qv[i] ^ hv[j]) >> 32));
              }
          };
          if (form == 2)
            inside_word([](uint32_t &best, uint32_t x) { tract_inside32_long(best, x); });
          else if (form == 1)
            inside_word([](uint32_t &best, uint32_t x) { tract_inside32_any(best, x); });
          else
            inside_word([](uint32_t &best, uint32_t x) { tract_inside32(best, x); });
        }
        continue;
      }
      common += tract_popc(m);
      if (m == ~0ull && chunk >= exact) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            tract_extend32(run[i][j], (uint32_t)(qv[i] ^ hv[j]));
            tract_extend32(run[i][j], (uint32_t)((qv[i] ^ hv[j]) >> 32));
          }
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tract_extend(run[i][j], (qv[i] ^ hv[j]) & m, m);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t q = qb + 2 * ty + i, s = (q0 + q) >> 1;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t h = hb + tx + 16 * j;
      uint32_t best = run[i][j].best;
      if (!all_exact && best == kRunFloor && q < nq && h < H) {  // no longer run: its exact length
        const uint64_t *const x = haps + (size_t)(q0 + q) * wn, *const y = haps + (size_t)h * wn;
        Tract t{0, 0, 0, 0};
        for (uint32_t w = 0; w < wn; ++w) {
          const uint64_t m = __ldg(mask + w);
          t = tract_join(t, tract_word((__ldg(x + w) ^ __ldg(y + w)) & m, m));
        }
        best = t.best;
      }
      const uint16_t d = (h >> 1) == s || h >= H ? kKnnExcluded : (uint16_t)(common - best);
      if (q < nq && h < pitch)  // excluded past H too
        dist[(size_t)q * pitch + h] = d;
      if (kSym)
        st[tx + 16 * j][2 * ty + i] = d;
    }
  }
  if (kSym) {
    __syncthreads();
    const uint32_t q = qb + (tid & 31u);
    for (uint32_t r = tid >> 5; r < kTractH; r += kDistThreads / 32) {
      // row h, column q: its own tile is not computed when it lies below the diagonal
      const uint32_t h = hb + r;
      if (h < H && q < nq && (qb & ~(kTractH - 1)) + kTractH <= (h & ~(kTractQ - 1)))
        dist[(size_t)h * pitch + q] = st[r][tid & 31u];
    }
  }
}

// The chunks of 8 words that knn_tract_dist_kernel takes exactly: the first where
// the words are six at most (`best` would rise inside most of them), where all tiles
// are computed and it is more than half of the words, and where fewer tiles than SMs
// leave a pair's chain of words to wait for; else none.  Tables in ms with none /
// one, typical haplotypes and (random ones), and in one pass over all tiles, as
// before either: 14,000 x 64 2.21 / 0.82 (1.73 / 0.84), 2.29; 14,000 x 384 3.33 / 3.10
// (5.33 / 3.13), 7.13; 14,000 x 448 3.44 / 3.53 (5.78 / 3.60), 7.95; 14,000 x 500 4.53 /
// 5.08 (8.29 / 7.14), 11.3; 14,000 x 1,024 5.31 / 6.21 (7.60 / 7.09), 15.9; all tiles,
// 24,000 x 1,024 30.0 / 35.4 (43.4 / 40.4), 45.3; few, 200 x 1,000 0.074 / 0.072 (0.104
// / 0.087), 0.098; 800 x 1,024 0.107 / 0.118 (0.130 / 0.121), 0.151.
constexpr uint32_t kTractExactWords = 6;
inline uint32_t tract_exact_chunks(uint32_t wn, bool sym, uint64_t tiles, int sms) {
  return wn <= kTractExactWords || (!sym && wn < 2 * kDistW) || tiles <= (uint64_t)sms ? 1 : 0;
}

// The neighbour lists of the samples s0 + blockIdx.x from their rows of
// distances (rows 2 i and 2 i + 1 of the chunk's i-th sample, `pitch` entries
// apart, those past H excluded): the `half` nearest to its first haplotype, then
// the `half` nearest to the second among those not taken, interleaved
// (KNN::ClusterHaps, kNN.cpp:170-206).  Where a wait of the distances' kernel ran
// out (kGemmTimeout in *error) they are not all there: the lists are filled with
// kKnnNoHap, which a generation refuses, and glp_finish reports the flag.
template <int kV>
__global__ void __launch_bounds__(kKnnThreads)
    knn_select_kernel(const uint16_t *__restrict__ dist, uint32_t pitch, uint32_t H, uint32_t s0,
                      uint32_t half, uint32_t dmax, const int *error,
                      uint32_t *__restrict__ neighbors) {
  __shared__ __align__(16) uint32_t keys[kKnnMaxHalf];
  __shared__ uint32_t chosen[2 * kKnnMaxHalf];
  __shared__ uint32_t taken[kKnnMaxHaps / 32 + 1];
  __shared__ uint32_t red[kKnnThreads / 32];
  static_assert(kSelectMost <= kKnnMaxHalf, "keys");
  const uint32_t tid = threadIdx.x;
  const uint16_t *const row = dist + (size_t)2 * blockIdx.x * pitch;
  uint32_t *const out = neighbors + (size_t)(s0 + blockIdx.x) * 2 * half;
  int flags = 0;
  for (uint32_t i = tid; i < (H + 31) / 32; i += kKnnThreads)
    taken[i] = 0;
  select_nearest<kV>(row, H, half, dmax, nullptr, keys, red, chosen, error, flags);
  for (uint32_t i = tid; i < half; i += kKnnThreads)
    if (chosen[i] < H)
      atomicOr(&taken[chosen[i] >> 5], 1u << (chosen[i] & 31u));
  __syncthreads();
  select_nearest<kV>(row + pitch, H, half, dmax, taken, keys, red, chosen + kKnnMaxHalf, nullptr,
                     flags);
  const bool failed = (flags & kGemmTimeout) != 0;
  for (uint32_t i = tid; i < half; i += kKnnThreads) {
    out[2 * i] = failed ? kKnnNoHap : chosen[i];
    out[2 * i + 1] = failed ? kKnnNoHap : chosen[kKnnMaxHalf + i];
  }
}

}  // namespace glp
