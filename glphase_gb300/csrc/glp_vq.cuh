// GL vector quantisation on the device: Lloyd training of the (homRef, het)
// codebook (GLVQ::BuildCodeBook / AssignPoints / UpdateCodeBook,
// src/glVQ.cpp:26-146) and the packing of codes into words
// (GLPack::GetPackedGLs, src/glPack.cpp:112-165).
//
// Points are the normalised pairs rr = g0 / s, het = g1 / s with
// s = (g0 + g1) + g2 (binary32) of the GL triples [N][S][3].  A point's code
// is the entry with the smallest distance, computed as GLVQHelper::
// EuclidianDist does (glVQ.hpp:23-30): the differences in binary32, squared
// and summed in binary64, then the square root; the first such entry wins.
//
// One training iteration = one vq_assign_kernel launch (assign every point
// and accumulate, per entry, the sums of rr and het, the count, and the
// total squared distance) + one vq_update_kernel launch (new entries).  Sums
// are binary64 in a fixed order, so they do not depend on scheduling: run r
// of block b holds points b*B + r + 256*j, j = 0..63 (B = 16,384), summed in
// j order; a block adds its 256 runs in r order; the update adds the blocks
// in b order.  (The reference sums in binary32 in point order; the host
// restatement in glphase_gb300/glpack.py uses this order.)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace glp {

constexpr int kVQMaxCodes = 16;
constexpr int kVQRun = 64;                          // points per thread
constexpr int kVQThreads = 256;                     // runs per block
constexpr uint32_t kVQBlock = kVQRun * kVQThreads;  // points per block

// a / s for the two quotients of a point, correctly rounded: with y the
// correctly rounded reciprocal of s and q within one unit of a / s, q + r y for
// the exact remainder r = a - s q rounds to RN(a / s) (P. Markstein, IA-64 and
// Elementary Functions, 2000, chapter 8); the first correction brings the
// product a y, which can be two units off, within one.  The operands' range keeps
// every remainder exact.  One reciprocal serves both quotients, and a zero
// numerator (frequent: probabilities clamped at 0) takes the same path.
// test_gpu_vq_quotient.py compares 10^10 quotients with the compiler's.
__device__ __forceinline__ float vq_quotient(float a, float s, float y) {
  const float q0 = __fmul_rn(a, y);
  const float q1 = __fmaf_rn(__fmaf_rn(-s, q0, a), y, q0);
  return __fmaf_rn(__fmaf_rn(-s, q1, a), y, q1);
}
__device__ __forceinline__ bool vq_quotient_ok(float a) {
  // +0, or of that range; the corrections would make -0 a +0
  return __float_as_uint(a) == 0u || (fabsf(a) >= 0x1p-80f && fabsf(a) <= 0x1p40f);
}
__device__ __forceinline__ void vq_normalise(float g0, float g1, float g2, float &rr,
                                             float &het) {
  const float s = __fadd_rn(__fadd_rn(g0, g1), g2);
  if (fabsf(s) >= 0x1p-30f && fabsf(s) <= 0x1p30f && vq_quotient_ok(g0) && vq_quotient_ok(g1)) {
    const float y = __frcp_rn(s);
    rr = vq_quotient(g0, s, y);
    het = vq_quotient(g1, s, y);
  } else {
    rr = __fdiv_rn(g0, s);
    het = __fdiv_rn(g1, s);
  }
}
__device__ __forceinline__ void vq_point(const float *__restrict__ gl, uint64_t p, float &rr,
                                         float &het) {
  vq_normalise(__ldg(gl + 3 * p), __ldg(gl + 3 * p + 1), __ldg(gl + 3 * p + 2), rr, het);
}

// Squared distance of EuclidianDist before the square root.
__device__ __forceinline__ double vq_d2(float cr, float ch, float rr, float het) {
  const double dx = (double)__fsub_rn(cr, rr), dy = (double)__fsub_rn(ch, het);
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
}

// Entry k of a kernel's codebook, which is padded to kVQMaxCodes entries with
// infinite ones (their distance is infinite, so they are never the nearest).
// An entry that repeats an earlier one never wins either, since the first
// smallest distance does: it is padded too, or every point near it would be a
// tie (few distinct GLs leave such entries: those without points move onto
// points).
__device__ __forceinline__ float2 vq_entry(const float2 *codebook, uint32_t K, uint32_t k) {
  const float inf = __int_as_float(0x7f800000);
  if (k >= K)
    return make_float2(inf, inf);
  const float2 e = codebook[k];
  for (uint32_t i = 0; i < k; ++i)
    if (codebook[i].x == e.x && codebook[i].y == e.y)
      return make_float2(inf, inf);
  return e;
}

// Nearest entry from the binary64 distances, among the entries whose binary32
// squared distance is at most `lim` (at least one is): the first with the smallest square root.  The square root is monotonic, so
// the first smallest squared distance is the answer unless an earlier entry's
// squared distance rounds to the same square root; those (within a few ulps)
// are checked with the root itself.
inline __device__ __noinline__ uint32_t vq_nearest_exact(const float2 *cb, uint32_t K, float rr,
                                                  float het, float lim) {
  uint32_t cand = 0;
  for (uint32_t k = 0; k < K; ++k) {
    const float dx = __fsub_rn(cb[k].x, rr), dy = __fsub_rn(cb[k].y, het);
    if (__fmaf_rn(dx, dx, __fmul_rn(dy, dy)) <= lim)
      cand |= 1u << k;
  }
  uint32_t kb = (uint32_t)__ffs(cand) - 1u;
  double best = vq_d2(cb[kb].x, cb[kb].y, rr, het);
  for (uint32_t m = cand & (cand - 1u); m; m &= m - 1u) {
    const uint32_t k = (uint32_t)__ffs(m) - 1u;
    const double d = vq_d2(cb[k].x, cb[k].y, rr, het);
    if (d < best) {
      best = d;
      kb = k;
    }
  }
  const double rb = __dsqrt_rn(best), near = best * (1.0 + 0x1p-48);
  for (uint32_t m = cand & ((1u << kb) - 1u); m; m &= m - 1u) {
    const uint32_t k = (uint32_t)__ffs(m) - 1u;
    const double d = vq_d2(cb[k].x, cb[k].y, rr, het);
    if (d <= near && __dsqrt_rn(d) == rb)
      return k;
  }
  return kb;
}

// Index of the first entry with the smallest sqrt(distance) for kVQPoints
// points at a time.  The differences are the reference's binary32 ones; their
// squared lengths are compared in binary32, whose relative error against the
// binary64 ones is below 2^-22 (underflow adds less than 2^-148): when the
// second smallest exceeds the smallest by more than a factor 1 + 2^-20 and
// 2^-100, every other entry's binary64 root is larger too and the smallest's
// index is the answer.  Otherwise (ties, near ties) the entries within that
// margin are compared in binary64.
// GB300 runs binary64 on two lanes an SM: with all 16 distances of a point in
// binary64 the assignment of 16.4 M points took 10.5 ms; with the binary32
// filter 0.36 ms, of which the binary64 pipe is busy half with the five
// operations a point that the sums need.
constexpr int kVQPoints = 4;
__device__ __forceinline__ void vq_nearest(const float2 *cb, uint32_t K, const float *rr,
                                           const float *het, uint32_t *code) {
  float d0[kVQPoints], m1[kVQPoints], m2[kVQPoints];
#pragma unroll
  for (int i = 0; i < kVQPoints; ++i) {
    const float dx = __fsub_rn(cb[0].x, rr[i]), dy = __fsub_rn(cb[0].y, het[i]);
    d0[i] = m1[i] = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
    m2[i] = __int_as_float(0x7f800000);
    code[i] = 0;
  }
#pragma unroll
  for (uint32_t k = 1; k < (uint32_t)kVQMaxCodes; ++k) {
    const float2 c = cb[k];
#pragma unroll
    for (int i = 0; i < kVQPoints; ++i) {
      const float dx = __fsub_rn(c.x, rr[i]), dy = __fsub_rn(c.y, het[i]);
      const float d = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
      code[i] = d < m1[i] ? k : code[i];
      m2[i] = fminf(m2[i], fmaxf(m1[i], d));
      m1[i] = fminf(m1[i], d);
    }
  }
#pragma unroll
  for (int i = 0; i < kVQPoints; ++i) {
    const float lim = __fmaf_rn(m1[i], 1.0f + 0x1p-20f, 0x1p-100f);
    if (d0[i] != d0[i])  // not a number: no entry compares below the first
      code[i] = 0;
    else if (!(m2[i] > lim))
      code[i] = vq_nearest_exact(cb, K, rr[i], het[i], lim);
  }
}

// A binary32 value as binary64 by integer operations (conversions run on the
// narrow binary64 pipe); zeros, subnormals, infinities and NaN convert.
inline __device__ __noinline__ double vq_widen_any(float x) { return (double)x; }
__device__ __forceinline__ double vq_widen(float x) {
  const uint32_t b = __float_as_uint(x), e = (b >> 23) & 0xffu;
  if (e - 1u >= 254u && x != 0.0f)  // subnormal, infinity or NaN
    return vq_widen_any(x);
  if (x == 0.0f)
    return __hiloint2double((int)b, 0);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)),
                          (int)(b << 29));
}

// Row stride of the per-run sums in shared memory: odd in doubles, so that the
// threads that add the runs of one sum each read distinct banks.
constexpr uint32_t kVQRow = kVQThreads + 1;

// Per block: sums[b][0..K) rr, [K..2K) het, [2K] squared distance (binary64),
// counts[b][0..K).  Dynamic shared memory: kVQRow * (2K + 1) doubles +
// kVQRow * K uint32.
__global__ void __launch_bounds__(kVQThreads)
    vq_assign_kernel(const float *__restrict__ gl, uint64_t P, const float2 *__restrict__ codebook,
                     uint32_t K, double *__restrict__ sums, uint32_t *__restrict__ counts) {
  extern __shared__ __align__(16) unsigned char vq_smem[];
  double *acc = reinterpret_cast<double *>(vq_smem);                    // [2K+1][kVQRow]
  uint32_t *cnt = reinterpret_cast<uint32_t *>(acc + (2 * K + 1) * kVQRow);  // [K][kVQRow]
  __shared__ float2 cb[kVQMaxCodes];
  const uint32_t t = threadIdx.x;
  if (t < (uint32_t)kVQMaxCodes)
    cb[t] = vq_entry(codebook, K, t);
  for (uint32_t i = 0; i < 2 * K + 1; ++i)
    acc[i * kVQRow + t] = 0.0;
  for (uint32_t k = 0; k < K; ++k)
    cnt[k * kVQRow + t] = 0;
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * kVQBlock + t;
  double var = 0.0;
  for (uint32_t j = 0; j < (uint32_t)kVQRun; j += kVQPoints) {
    float rr[kVQPoints], het[kVQPoints];
    uint32_t code[kVQPoints];
    const uint64_t p0 = base + (uint64_t)j * kVQThreads;
    if (p0 >= P)
      break;
#pragma unroll
    for (int i = 0; i < kVQPoints; ++i)  // points past the end repeat the first, unused
      vq_point(gl, p0 + (uint64_t)i * kVQThreads < P ? p0 + (uint64_t)i * kVQThreads : p0, rr[i],
               het[i]);
    vq_nearest(cb, K, rr, het, code);
#pragma unroll
    for (int i = 0; i < kVQPoints; ++i) {
      if (p0 + (uint64_t)i * kVQThreads >= P)
        break;
      const uint32_t k = code[i];
      double *a = acc + k * kVQRow + t;
      *a = __dadd_rn(*a, vq_widen(rr[i]));
      a += K * kVQRow;
      *a = __dadd_rn(*a, vq_widen(het[i]));
      cnt[k * kVQRow + t] += 1;
      // AssignPoints' term: the differences point - entry in binary32, squared
      // and summed in binary64 (a binary32 value's square is exact there, so
      // the fused form rounds once, as the two products and the sum do)
      const double dx = vq_widen(__fsub_rn(rr[i], cb[k].x)),
                   dy = vq_widen(__fsub_rn(het[i], cb[k].y));
      var = __dadd_rn(var, __fma_rn(dx, dx, __dmul_rn(dy, dy)));
    }
  }
  acc[2 * K * kVQRow + t] = var;
  __syncthreads();
  // runs in r order: one thread per sum
  if (t < 2 * K + 1) {
    double s = 0.0;
    const double *row = acc + t * kVQRow;
#pragma unroll 8
    for (uint32_t r = 0; r < (uint32_t)kVQThreads; ++r)
      s = __dadd_rn(s, row[r]);
    sums[(uint64_t)blockIdx.x * (2 * K + 1) + t] = s;
  } else if (t >= 64 && t < 64 + K) {
    uint32_t c = 0;
    const uint32_t *row = cnt + (t - 64) * kVQRow;
#pragma unroll 8
    for (uint32_t r = 0; r < (uint32_t)kVQThreads; ++r)
      c += row[r];
    counts[(uint64_t)blockIdx.x * K + t - 64] = c;
  }
}

// SplitMix64 (Steele, Lea, Flood 2014): the point an entry with no points
// moves to, for training iteration `it` (UpdateCodeBook draws a random point
// there, glVQ.cpp:127-133).
__host__ __device__ inline uint64_t vq_splitmix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
// Shared memory of vq_assign_kernel for K entries.
__host__ __device__ constexpr size_t vq_assign_smem(uint32_t K) {
  return (size_t)kVQRow * ((2 * K + 1) * sizeof(double) + K * sizeof(uint32_t));
}

__host__ __device__ inline uint64_t vq_empty_point(uint64_t seed, uint32_t it, uint32_t k,
                                                   uint64_t P) {
  return vq_splitmix64(seed ^ (((uint64_t)it << 16) | k)) % P;
}

// New entries from the block sums (blocks in b order): mean of the points
// of an entry rounded to binary32, or an empty entry moved onto a point.
// out_var = the total squared distance of the assignment the sums came from.
// One block of kVQUpdThreads threads: the sums of kVQUpdBlocks blocks at a time
// go through shared memory (the next ones already on their way), where one
// thread a sum adds them; what is left is the chain of binary64 additions
// (1,001 blocks of 16.4 M points: 147 us with each addend loaded in the chain,
// 58 us this way).
constexpr uint32_t kVQUpdThreads = 256, kVQUpdBlocks = 32;
__global__ void __launch_bounds__(kVQUpdThreads)
    vq_update_kernel(const float *__restrict__ gl, uint64_t P, uint32_t nblocks,
                     const double *__restrict__ sums, const uint32_t *__restrict__ counts,
                     uint32_t K, uint64_t seed, uint32_t it, float2 *__restrict__ codebook,
                     double *__restrict__ out_var) {
  constexpr uint32_t kMost = kVQUpdBlocks * (2 * kVQMaxCodes + 1);
  constexpr uint32_t kPer = (kMost + kVQUpdThreads - 1) / kVQUpdThreads;
  __shared__ double part[2][kMost];
  __shared__ double tot[2 * kVQMaxCodes + 1];
  __shared__ unsigned long long num[kVQMaxCodes];
  const uint32_t t = threadIdx.x, W = 2 * K + 1;
  const uint64_t all = (uint64_t)nblocks * W;
  const uint32_t span = kVQUpdBlocks * W;
  double next[kPer];
  auto fetch = [&](uint64_t from) {
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
      const uint32_t o = t + i * kVQUpdThreads;
      next[i] = (o < span && from + o < all) ? sums[from + o] : 0.0;
    }
  };
  fetch(0);
  __syncthreads();
  double s = 0.0;
  uint32_t buf = 0;
  for (uint32_t b0 = 0; b0 < nblocks; b0 += kVQUpdBlocks, buf ^= 1) {
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
      const uint32_t o = t + i * kVQUpdThreads;
      if (o < span)
        part[buf][o] = next[i];
    }
    fetch((uint64_t)(b0 + kVQUpdBlocks) * W);
    __syncthreads();  // the other buffer is refilled only after the next barrier
    if (t < W) {
      const uint32_t n = min(kVQUpdBlocks, nblocks - b0);
      if (n == kVQUpdBlocks) {
#pragma unroll
        for (uint32_t b = 0; b < kVQUpdBlocks; ++b)
          s = __dadd_rn(s, part[buf][b * W + t]);
      } else {
        for (uint32_t b = 0; b < n; ++b)
          s = __dadd_rn(s, part[buf][b * W + t]);
      }
    }
  }
  if (t < W)
    tot[t] = s;
  for (uint32_t k = t >> 5; k < K; k += kVQUpdThreads / 32) {
    unsigned long long c = 0;
#pragma unroll 8
    for (uint32_t b = t & 31u; b < nblocks; b += 32)
      c += counts[(uint64_t)b * K + k];
    for (int o = 16; o; o >>= 1)
      c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((t & 31u) == 0)
      num[k] = c;
  }
  __syncthreads();
  if (t == 0)
    *out_var = tot[2 * K];
  if (t < K) {
    float2 e;
    if (num[t] > 0) {
      e.x = (float)__ddiv_rn(tot[t], (double)num[t]);
      e.y = (float)__ddiv_rn(tot[K + t], (double)num[t]);
    } else {
      vq_point(gl, vq_empty_point(seed, it, t, P), e.x, e.y);
    }
    codebook[t] = e;
  }
}

// Codes of sites w*per .. w*per+per-1 of sample n packed into one word,
// first site in the most significant bits; sites past S use the array's
// first GL (glPack.cpp:147-149).  packed is [ceil(S/per)][N].
struct VQBook {
  float2 e[kVQMaxCodes];
};

// A block takes 32 samples x 64 sites, a warp four samples at a time: lane l
// codes site l of each half, the lanes of a word join their codes, and the
// words leave through shared memory, a word's 32 samples together.  Bound by
// the binary32 distances' instructions and the loads' latency (2,000 x 8,192
// sites: 0.28 ms; 9.47 ms with one word a thread and binary64 distances).
constexpr uint32_t kVQPackSamples = 32, kVQPackSites = 64, kVQPackThreads = 256;
static_assert(kVQPackSamples == kVQPoints * kVQPackThreads / 32, "one pass over the samples");
__global__ void __launch_bounds__(kVQPackThreads)
    vq_pack_kernel(const float *__restrict__ gl, uint32_t N, uint32_t S, const VQBook book,
                   uint32_t K, uint32_t bits, uint32_t *__restrict__ packed) {
  __shared__ float2 cb[kVQMaxCodes];
  __shared__ uint32_t words[kVQPackSites / 4][kVQPackSamples + 1];  // at least 4 sites a word
  const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31u;
  if (t < (uint32_t)kVQMaxCodes)
    cb[t] = vq_entry(book.e, K, t);
  const uint32_t tiles = (N + kVQPackSamples - 1) / kVQPackSamples;  // of samples
  const uint32_t n0 = blockIdx.x % tiles * kVQPackSamples,
                 m0 = blockIdx.x / tiles * kVQPackSites;
  const uint32_t per = 32u / bits, nw = (S + per - 1) / per, wt = kVQPackSites / per;
  __syncthreads();
#pragma unroll
  for (uint32_t h = 0; h < kVQPackSites; h += 32) {
    const uint32_t m = m0 + h + lane;
    float rr[kVQPoints], het[kVQPoints];
    uint32_t code[kVQPoints];
#pragma unroll
    for (int i = 0; i < kVQPoints; ++i) {
      const uint32_t n = n0 + warp * kVQPoints + i;
      // sites past S (and idle samples) take the array's first GL
      vq_point(gl, (n < N && m < S) ? (uint64_t)n * S + m : 0, rr[i], het[i]);
    }
    vq_nearest(cb, K, rr, het, code);
#pragma unroll
    for (int i = 0; i < kVQPoints; ++i) {
      uint32_t w = code[i] << (32u - bits * (lane % per + 1));
      for (uint32_t o = 1; o < per; o <<= 1)
        w |= __shfl_xor_sync(0xffffffffu, w, o);
      if (lane % per == 0)
        words[(h + lane) / per][warp * kVQPoints + i] = w;
    }
  }
  __syncthreads();
  for (uint32_t wi = warp; wi < wt; wi += kVQPackThreads / 32) {
    const uint32_t w = m0 / per + wi, n = n0 + lane;
    if (w < nw && n < N)
      packed[(uint64_t)w * N + n] = words[wi][lane];
  }
}

}  // namespace glp
