// glp_tally.cuh -- per-site allele tallies of the sampling generations on the
// device: Impute::replace (src/impute.cpp:564-595) and Impute::result
// (src/impute.cpp:599-613).
//
// replace: for sample I with current haplotypes oa, ob and running tallies
// ha, hb ([2N][S] uint32), count sis = sum over alt sites of oa of ha plus
// alt sites of ob of hb, and tra the crossed sum; then add oa to ha and ob to
// hb when sis > tra, else crossed.  Integer arithmetic: bit-exact.
// One CTA per sample; the two sums are block reductions in 32-bit arithmetic, as
// the reference's unsigned sums are.
//
// Bound: HBM, two rows read and written once: each thread keeps its share of
// both rows (kHold vectors of four sites) in registers between the sums and the
// update, so that the rows are read once (with a second read, from L2 at best,
// 10,000 x 4,096 took 163 us; this form 113, 5.8 TB/s).  The rows' sums are
// separate, so where S is no multiple of 4 each row has vectors of its own, from
// its first aligned address, and up to six single sites at its ends (4,000 x 4,097:
// 67.6 us; 98 by single sites, 84 with the rows read twice).  Short rows are bound
// by what a block costs: few threads and few registers (8,000 x 101: 8.2 us; 28.8
// with the registers of the longest rows, 10.3 before rows were held).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace glp {

// Vectors a thread holds and threads a block for S sites: one where 128 threads
// cover a row, two up to 256, else four with up to 1,024 threads; rows beyond
// 16,384 sites are read twice past that.
inline int tally_hold(uint32_t S) { return S <= 512 ? 1 : S <= 1024 ? 2 : 4; }
inline uint32_t tally_threads(uint32_t S) {
  uint32_t t = S <= 512 ? 32 : 128;
  while (t < 1024 && (uint64_t)t * 4 * tally_hold(S) < S)
    t *= 2;
  return t;
}

// The alleles of the sites m .. m + 3 of a row of words; kAligned: m is a multiple
// of 4.
template <bool kAligned>
__device__ __forceinline__ uint32_t tally_bits(const uint64_t *__restrict__ row, uint32_t m) {
  const uint32_t w = m >> 6, sh = m & 63u;
  uint64_t x = __ldg(row + w) >> sh;
  if (!kAligned && sh > 60u)
    x |= __ldg(row + w + 1) << (64u - sh);
  return (uint32_t)x;
}
__device__ __forceinline__ uint32_t &tally_at(uint4 &v, int i) {
  return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}
// Sum of the tallies of v at alternative alleles.
__device__ __forceinline__ uint32_t tally_sum(uint4 &v, uint32_t bits) {
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    s += (0u - ((bits >> i) & 1u)) & tally_at(v, i);
  return s;
}

// kAligned: both rows start on 16 bytes and S is a multiple of 4.
template <int kHold, bool kAligned>
__global__ void __launch_bounds__(kHold == 4 ? 1024 : 128)
    replace_kernel(const uint64_t *__restrict__ haps, uint32_t N, uint32_t S, uint32_t wn,
                   uint32_t *__restrict__ hsum) {
  const uint32_t I = blockIdx.x, tid = threadIdx.x, step = blockDim.x;
  const uint64_t *const oa = haps + (size_t)2 * I * wn, *const ob = oa + wn;
  uint32_t *const ha = hsum + (size_t)2 * I * S, *const hb = ha + S;
  // the sites before a row's first vector, and its vectors
  auto first = [&](const uint32_t *row) {
    return kAligned ? 0u : min(S, (0u - (uint32_t)((uintptr_t)row >> 2)) & 3u);
  };
  const uint32_t fa = first(ha), fb = first(hb), na = (S - fa) / 4, nb = (S - fb) / 4;
  uint4 *const va = reinterpret_cast<uint4 *>(ha + fa),
        *const vb = reinterpret_cast<uint4 *>(hb + fb);
  uint4 x[kHold], y[kHold];
#pragma unroll
  for (int k = 0; k < kHold; ++k) {
    const uint32_t v = tid + k * step;
    if (v < na)
      x[k] = __ldcs(va + v);
    if (v < nb)
      y[k] = __ldcs(vb + v);
  }
  // the single sites: threads 0 .. 7 row a's, 8 .. 15 row b's
  uint32_t *one = nullptr;
  uint32_t e = 0, ea = 0, eb = 0;  // its tally and alleles
  if (!kAligned && tid < 16) {
    const uint32_t f = tid < 8 ? fa : fb, n = tid < 8 ? na : nb, i = tid & 7u,
                   m = i < f ? i : i + 4 * n;
    if (m < S && i < S - 4 * n) {
      one = (tid < 8 ? ha : hb) + m;
      e = *one;
      ea = (uint32_t)(__ldg(oa + (m >> 6)) >> (m & 63u)) & 1u;
      eb = (uint32_t)(__ldg(ob + (m >> 6)) >> (m & 63u)) & 1u;
    }
  }
  uint32_t sis = (tid < 8 ? ea : eb) * e, tra = (tid < 8 ? eb : ea) * e;
  auto sum_a = [&](uint4 &t, uint32_t v) {
    sis += tally_sum(t, tally_bits<kAligned>(oa, fa + 4 * v));
    tra += tally_sum(t, tally_bits<kAligned>(ob, fa + 4 * v));
  };
  auto sum_b = [&](uint4 &t, uint32_t v) {
    sis += tally_sum(t, tally_bits<kAligned>(ob, fb + 4 * v));
    tra += tally_sum(t, tally_bits<kAligned>(oa, fb + 4 * v));
  };
#pragma unroll
  for (int k = 0; k < kHold; ++k) {
    const uint32_t v = tid + k * step;
    if (v < na)
      sum_a(x[k], v);
    if (v < nb)
      sum_b(y[k], v);
  }
  for (uint32_t v = tid + kHold * step; v < max(na, nb); v += step) {
    uint4 t;
    if (v < na)
      sum_a(t = va[v], v);
    if (v < nb)
      sum_b(t = vb[v], v);
  }
  sis = __reduce_add_sync(0xffffffffu, sis);
  tra = __reduce_add_sync(0xffffffffu, tra);
  if (step > 32) {
    __shared__ uint32_t r_s[32], r_t[32];
    if ((tid & 31u) == 0) {
      r_s[tid >> 5] = sis;
      r_t[tid >> 5] = tra;
    }
    __syncthreads();
    const uint32_t lane = tid & 31u, warps = step >> 5;
    sis = __reduce_add_sync(0xffffffffu, lane < warps ? r_s[lane] : 0u);
    tra = __reduce_add_sync(0xffffffffu, lane < warps ? r_t[lane] : 0u);
  }
  const bool keep = sis > tra;
  const uint64_t *const ka = keep ? oa : ob, *const kb = keep ? ob : oa;
  auto add = [&](uint4 &t, const uint64_t *row, uint32_t m) {
    const uint32_t b = tally_bits<kAligned>(row, m);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      tally_at(t, i) += (b >> i) & 1u;
  };
#pragma unroll
  for (int k = 0; k < kHold; ++k) {
    const uint32_t v = tid + k * step;
    if (v < na) {
      add(x[k], ka, fa + 4 * v);
      va[v] = x[k];
    }
    if (v < nb) {
      add(y[k], kb, fb + 4 * v);
      vb[v] = y[k];
    }
  }
  for (uint32_t v = tid + kHold * step; v < max(na, nb); v += step) {
    uint4 t;
    if (v < na) {
      add(t = va[v], ka, fa + 4 * v);
      va[v] = t;
    }
    if (v < nb) {
      add(t = vb[v], kb, fb + 4 * v);
      vb[v] = t;
    }
  }
  if (!kAligned && one)
    *one = e + ((tid < 8) == keep ? ea : eb);
}

// result: prob_out[m][2i + h] = hsum[(2i + h)][m] * (float)(1 / sn)
// (impute.cpp:599-613), binary32.  Tiles of 64 haplotypes x 64 sites turned in
// shared memory, so that both sides move 256 bytes a row.  Bound: HBM (10,000 x
// 4,096: 388 us with one thread an entry reading down a column, 114 us, 5.8 TB/s).
// Few entries, whose columns stay in L1, take one thread each, without a tile's
// two trips: 500 x 3 2.9 us (4.2 by tiles), 60 x 255 3.8 (4.2), level at 2^18 entries.
constexpr uint64_t kResultSmall = (uint64_t)1 << 18;
constexpr uint32_t kResultSmallThreads = 256;
__global__ void __launch_bounds__(kResultSmallThreads)
    result_small_kernel(const uint32_t *__restrict__ hsum, uint32_t H, uint32_t S, float norm,
                        float *__restrict__ prob_out) {
  const uint32_t i = blockIdx.x * kResultSmallThreads + threadIdx.x, m = i / H, h = i % H;
  if (m < S)
    prob_out[i] = (float)__ldg(hsum + h * S + m) * norm;
}

constexpr uint32_t kResultTile = 64, kResultThreads = 256;
__global__ void __launch_bounds__(kResultThreads)
    result_kernel(const uint32_t *__restrict__ hsum, uint32_t N, uint32_t S, uint32_t site_tiles,
                  float norm, float *__restrict__ prob_out) {
  __shared__ uint32_t tile[kResultTile][kResultTile + 1];
  const size_t H = (size_t)2 * N;
  const uint32_t m0 = blockIdx.x % site_tiles * kResultTile;
  const size_t h0 = (size_t)(blockIdx.x / site_tiles) * kResultTile;
  const uint32_t c = threadIdx.x % kResultTile, r0 = threadIdx.x / kResultTile;
#pragma unroll 4
  for (uint32_t r = r0; r < kResultTile; r += kResultThreads / kResultTile)
    if (h0 + r < H && m0 + c < S)
      tile[r][c] = __ldcs(hsum + (h0 + r) * S + m0 + c);
  __syncthreads();
#pragma unroll 4
  for (uint32_t r = r0; r < kResultTile; r += kResultThreads / kResultTile)
    if (m0 + r < S && h0 + c < H)
      __stcs(prob_out + (size_t)(m0 + r) * H + h0 + c, (float)tile[c][r] * norm);
}

}  // namespace glp
