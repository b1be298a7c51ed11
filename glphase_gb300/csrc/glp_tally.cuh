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
// both rows (kHold loads of kW consecutive sites) in registers between the sums
// and the update, so that the rows are read once (with a second read, from L2
// at best, 10,000 x 4,096 took 163 us; this form 117, 5.6 TB/s).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace glp {

template <int kW>
struct TallyLoad;
template <>
struct TallyLoad<4> {  // rows of whole, aligned 16-byte vectors
  using T = uint4;
  static constexpr int kHold = 4;
  static __device__ __forceinline__ uint32_t &at(uint4 &v, int i) {
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
  }
};
template <>
struct TallyLoad<1> {
  using T = uint32_t;
  static constexpr int kHold = 16;
  static __device__ __forceinline__ uint32_t &at(uint32_t &v, int) { return v; }
};

// Threads a block for S sites: enough that the registers hold the rows, up to
// 1,024 (longer rows are read twice past kHold loads a thread).
inline uint32_t tally_threads(uint32_t S) {
  uint32_t t = 128;
  while (t < 1024 && t * 16 < S)
    t *= 2;
  return t;
}

template <int kW>
__global__ void __launch_bounds__(1024)
    replace_kernel(const uint64_t *__restrict__ haps, uint32_t N, uint32_t S, uint32_t wn,
                   uint32_t *__restrict__ hsum) {
  using L = TallyLoad<kW>;
  using T = typename L::T;
  const uint32_t I = blockIdx.x, tid = threadIdx.x, step = blockDim.x, nv = S / kW;
  const uint64_t *const oa = haps + (size_t)2 * I * wn, *const ob = oa + wn;
  T *const ha = reinterpret_cast<T *>(hsum + (size_t)2 * I * S),
    *const hb = reinterpret_cast<T *>(hsum + (size_t)2 * I * S + S);
  // the alleles of load v: kW bits a haplotype
  auto bits = [&](const uint64_t *row, uint32_t v) {
    const uint32_t m = v * kW;
    return (uint32_t)(__ldg(row + (m >> 6)) >> (m & 63u));
  };
  uint32_t sis = 0, tra = 0;
  auto sums = [&](T &x, T &y, uint32_t a, uint32_t b) {
#pragma unroll
    for (int i = 0; i < kW; ++i) {
      const uint32_t xs = L::at(x, i), ys = L::at(y, i);
      const uint32_t am = 0u - ((a >> i) & 1u), bm = 0u - ((b >> i) & 1u);
      sis += (am & xs) + (bm & ys);
      tra += (am & ys) + (bm & xs);
    }
  };
  T x[L::kHold], y[L::kHold];
#pragma unroll
  for (int k = 0; k < L::kHold; ++k) {
    const uint32_t v = tid + k * step;
    if (v < nv) {
      x[k] = __ldcs(ha + v);
      y[k] = __ldcs(hb + v);
    }
  }
#pragma unroll
  for (int k = 0; k < L::kHold; ++k) {
    const uint32_t v = tid + k * step;
    if (v < nv)
      sums(x[k], y[k], bits(oa, v), bits(ob, v));
  }
  for (uint32_t v = tid + L::kHold * step; v < nv; v += step) {
    T xv = ha[v], yv = hb[v];
    sums(xv, yv, bits(oa, v), bits(ob, v));
  }
  __shared__ uint32_t r_s[32], r_t[32];
  sis = __reduce_add_sync(0xffffffffu, sis);
  tra = __reduce_add_sync(0xffffffffu, tra);
  if ((tid & 31u) == 0) {
    r_s[tid >> 5] = sis;
    r_t[tid >> 5] = tra;
  }
  __syncthreads();
  const uint32_t lane = tid & 31u, warps = step >> 5;
  sis = __reduce_add_sync(0xffffffffu, lane < warps ? r_s[lane] : 0u);
  tra = __reduce_add_sync(0xffffffffu, lane < warps ? r_t[lane] : 0u);
  const bool keep = sis > tra;
  const uint64_t *const ka = keep ? oa : ob, *const kb = keep ? ob : oa;
  auto add = [&](T &xv, T &yv, uint32_t v) {
    const uint32_t a = bits(ka, v), b = bits(kb, v);
#pragma unroll
    for (int i = 0; i < kW; ++i) {
      L::at(xv, i) += (a >> i) & 1u;
      L::at(yv, i) += (b >> i) & 1u;
    }
  };
#pragma unroll
  for (int k = 0; k < L::kHold; ++k) {
    const uint32_t v = tid + k * step;
    if (v < nv) {
      add(x[k], y[k], v);
      ha[v] = x[k];
      hb[v] = y[k];
    }
  }
  for (uint32_t v = tid + L::kHold * step; v < nv; v += step) {
    T xv = ha[v], yv = hb[v];
    add(xv, yv, v);
    ha[v] = xv;
    hb[v] = yv;
  }
}

// result: prob_out[m][2i + h] = hsum[(2i + h)][m] * (float)(1 / sn)
// (impute.cpp:599-613), binary32.  Tiles of 64 haplotypes x 64 sites turned in
// shared memory, so that both sides move 256 bytes a row.  Bound: HBM (10,000 x
// 4,096: 388 us with one thread an entry reading down a column, 114 us, 5.8 TB/s).
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
