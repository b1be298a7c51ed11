// glp_knn_gemm.cuh -- Hamming distances of the kNN tables as a matrix product on
// the tensor cores (haplotype.cpp:35-60 over the common sites of kNN.cpp:216-257).
//
// A haplotype's common sites become +1 (alternative allele) and -1 in 8 bits
// (e4m3), the other sites 0, so that for two of them
//   product = agreements - disagreements,  distance = (sites - product) / 2.
// Products of +-1 and sums below 2^16 are exact in the binary32 accumulators.
//
// One CTA computes 128 query haplotypes x 256 haplotypes: K in steps of 128 sites
// (one 128-byte swizzled row), each step's operands staged by TMA, four
// tcgen05.mma a step from one thread into 256 TMEM columns, read back by four
// warps.  Two CTAs share an SM, so one's epilogue runs beside the other's products.
// Distances are symmetric: over the whole panel only the tiles on and above the
// diagonal are computed, and written twice.
//
// What bounds it: a step feeds 48 KB of operands to 512 cycles of products, 96
// bytes a cycle and SM from L2.  20,000 haplotypes x 4,096 sites: 0.72 ms (2.3
// PFLOP/s of products computed); 10.5 ms as population counts, which ran at 97 % of
// their pipe.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "glp_knn.cuh"

namespace glp {

constexpr uint32_t kGemmM = 128, kGemmN = 256, kGemmK = kKnnOperandStep;  // sites = bytes
constexpr uint32_t kGemmStages = 2;
constexpr uint32_t kGemmABytes = kGemmM * kGemmK, kGemmBBytes = kGemmN * kGemmK;
constexpr uint32_t kGemmStageBytes = kGemmABytes + kGemmBBytes;
constexpr int kGemmThreads = 192;  // producer, product and four epilogue warps
constexpr size_t kGemmSmem = 1024 + (size_t)kGemmStages * kGemmStageBytes;
constexpr uint64_t kGemmWaitNs = 2000000000ull;  // after which a wait gives up

// Rows h0 .. h0 + rows - 1 of the panel as operand rows of `pitch` bytes, 16
// sites a thread.  Bound: the stores (20,000 x 4,096: 82 MB).
__global__ void __launch_bounds__(256)
    knn_expand_kernel(const uint64_t *__restrict__ haps, uint32_t h0, uint32_t rows, uint32_t wn,
                      const uint64_t *__restrict__ mask, uint32_t pitch, uint4 *__restrict__ out) {
  const uint32_t per = pitch / 16;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (uint64_t)rows * per)
    return;
  const uint32_t r = (uint32_t)(i / per), g = (uint32_t)(i % per), w = g >> 2,
                 sh = 16 * (g & 3u);
  uint32_t bits = 0, keep = 0;
  if (w < wn) {
    bits = (uint32_t)(__ldg(haps + (size_t)(h0 + r) * wn + w) >> sh) & 0xffffu;
    keep = (uint32_t)(__ldg(mask + w) >> sh) & 0xffffu;
  }
  uint32_t o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    // four bits to the low bits of four bytes
    const uint32_t kb = ((keep >> (4 * k)) & 15u) * 0x00204081u & 0x01010101u;
    const uint32_t zb = (((keep & ~bits) >> (4 * k)) & 15u) * 0x00204081u & 0x01010101u;
    o[k] = kb * 0x38u | zb << 7;  // e4m3: 0x38 = 1, the sign in bit 7
  }
  out[i] = make_uint4(o[0], o[1], o[2], o[3]);
}

// Number of common sites.
__global__ void knn_sites_kernel(const uint64_t *__restrict__ mask, uint32_t wn,
                                 uint32_t *__restrict__ sites) {
  uint32_t n = 0;
  for (uint32_t w = threadIdx.x; w < wn; w += 32)
    n += (uint32_t)__popcll(__ldg(mask + w));
  n = __reduce_add_sync(0xffffffffu, n);
  if (threadIdx.x == 0)
    *sites = n;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase of parity `parity`; false once `limit` nanoseconds have passed.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          uint64_t limit = kGemmWaitNs) {
  uint64_t until = 0;
  for (uint32_t n = 0;; ++n) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done)
      return true;
    if ((n & 63u) == 63u) {
      const uint64_t now = global_ns();
      if (!until)
        until = now + limit;
      else if (now > until)
        return false;
    }
  }
}
__device__ __forceinline__ void tma_load(const CUtensorMap *map, void *dst, uint64_t *bar, int x,
                                         int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(smem_addr(bar)), "r"(x), "r"(y)
      : "memory");
}
// Shared-memory descriptor of a K-major operand with 128-byte swizzle: rows of
// 128 bytes, groups of 8 rows 1,024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// Distances of the queries' operand rows [a0, a0 + nq) against the rows [b0, b0
// + nh) of the haplotypes' operand; row r of the output is query q0 + r, column c
// haplotype c (h0 + the tile's column), up to the pitch.  A sample's own two and
// columns from H on are marked excluded.  grid: tiles of 128 queries (x) by
// tiles of 256 haplotypes (y).  kSym: queries and haplotypes are the whole panel;
// tiles below the diagonal are not computed, their distances are written with
// the tiles above it, transposed.
template <bool kSym>
__global__ void __launch_bounds__(kGemmThreads)
    knn_gemm_kernel(const __grid_constant__ CUtensorMap amap,
                    const __grid_constant__ CUtensorMap bmap, uint32_t a0, uint32_t b0,
                    uint32_t nq, uint32_t nh, uint32_t q0, uint32_t h0, uint32_t H,
                    uint32_t steps, const uint32_t *__restrict__ sites, uint32_t pitch,
                    uint16_t *__restrict__ dist, int *__restrict__ error) {
  const uint32_t tm = blockIdx.x, tn = blockIdx.y;
  if (kSym && 2 * tn + 1 < tm)
    return;
  extern __shared__ unsigned char gemm_smem_raw[];
  unsigned char *const smem = reinterpret_cast<unsigned char *>(
      ((uintptr_t)gemm_smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kGemmStages], empty[kGemmStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kGemmStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&tmem_base)),
                 "r"(kGemmN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  if (warp == 0 && lane == 0) {
    uint32_t issued = 0;
    bool ok = true;
    for (; issued < steps; ++issued) {
      const uint32_t s = issued % kGemmStages, round = issued / kGemmStages;
      if (round && !(ok = mbar_wait(&empty[s], (round - 1) & 1u)))
        break;
      unsigned char *const a = smem + s * kGemmStageBytes, *const b = a + kGemmABytes;
      const int x = (int)(issued * kGemmK);
      mbar_expect(&full[s], kGemmStageBytes);
      tma_load(&amap, a, &full[s], x, (int)(a0 + tm * kGemmM));
      tma_load(&bmap, b, &full[s], x, (int)(b0 + tn * kGemmN));
      tma_load(&bmap, b + kGemmBBytes / 2, &full[s], x, (int)(b0 + tn * kGemmN + kGemmN / 2));
    }
    if (!ok) {  // the copies in flight end before the block does
      failed = 1;
      for (uint32_t k = issued > kGemmStages ? issued - kGemmStages : 0; k < issued; ++k)
        mbar_wait(&full[k % kGemmStages], (k / kGemmStages) & 1u);
    }
  } else if (warp == 1 && lane == 0) {
    // kind::f8f6f4, binary32 accumulators, both operands e4m3 and K-major
    constexpr uint32_t idesc = 1u << 4 | (kGemmN >> 3) << 17 | (kGemmM >> 4) << 24;
    bool ok = true;
    for (uint32_t k = 0; k < steps && ok; ++k) {
      const uint32_t s = k % kGemmStages;
      ok = mbar_wait(&full[s], (k / kGemmStages) & 1u);
      if (!ok)
        break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a = smem_addr(smem) + s * kGemmStageBytes;
      const uint64_t da = umma_desc(a), db = umma_desc(a + kGemmABytes);
#pragma unroll
      for (uint32_t j = 0; j < kGemmK / 32; ++j) {  // 32 sites a product: 32 bytes on
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(da + 2 * j), "l"(db + 2 * j), "r"(idesc), "r"(k | j)
            : "memory");
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_addr(&empty[s]))
          : "memory");
    }
    if (!ok)
      failed = 1;
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_addr(&done))
        : "memory");
  } else if (warp >= 2) {
    if (!__all_sync(0xffffffffu, mbar_wait(&done, 0))) {
      if (lane == 0)
        failed = 1;
    } else {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t quarter = warp & 3u;  // the TMEM lanes a warp may read
      const uint32_t r = tm * kGemmM + 32 * quarter + lane, q = q0 + r;
      const float half_sites = 0.5f * (float)__ldg(sites);
      const bool own = q0 + tm * kGemmM < h0 + tn * kGemmN + kGemmN &&
                       h0 + tn * kGemmN < q0 + tm * kGemmM + kGemmM;
#pragma unroll 1
      for (uint32_t c0 = 0; c0 < kGemmN; c0 += 32) {
        const uint32_t c = tn * kGemmN + c0;
        uint32_t acc[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
            "[%32];\n\ttcgen05.wait::ld.sync.aligned;"
            : "=r"(acc[0]), "=r"(acc[1]), "=r"(acc[2]), "=r"(acc[3]), "=r"(acc[4]), "=r"(acc[5]),
              "=r"(acc[6]), "=r"(acc[7]), "=r"(acc[8]), "=r"(acc[9]), "=r"(acc[10]),
              "=r"(acc[11]), "=r"(acc[12]), "=r"(acc[13]), "=r"(acc[14]), "=r"(acc[15]),
              "=r"(acc[16]), "=r"(acc[17]), "=r"(acc[18]), "=r"(acc[19]), "=r"(acc[20]),
              "=r"(acc[21]), "=r"(acc[22]), "=r"(acc[23]), "=r"(acc[24]), "=r"(acc[25]),
              "=r"(acc[26]), "=r"(acc[27]), "=r"(acc[28]), "=r"(acc[29]), "=r"(acc[30]),
              "=r"(acc[31])
            : "r"(tmem + (32 * quarter << 16) + c0)
            : "memory");
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          // (sites - product) / 2, an integer below 2^16, in the low bits
          const float d = fmaf(__uint_as_float(acc[j]), -0.5f, half_sites);
          acc[j] = __float_as_uint(d + 8388608.0f) & 0xffffu;
        }
        if (own || h0 + c + 32 > H) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (((h0 + c + j) >> 1) == (q >> 1) || h0 + c + j >= H)
              acc[j] = kKnnExcluded;
        }
        if (r < nq && h0 + c < pitch) {  // whole groups of 32 columns: pitch is a multiple of 128
          uint4 *const to = reinterpret_cast<uint4 *>(dist + (size_t)r * pitch + h0 + c);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            __stcs(to + j, make_uint4(acc[8 * j] | acc[8 * j + 1] << 16,
                                      acc[8 * j + 2] | acc[8 * j + 3] << 16,
                                      acc[8 * j + 4] | acc[8 * j + 5] << 16,
                                      acc[8 * j + 6] | acc[8 * j + 7] << 16));
        }
        // column block c / 128 against row block tm: the transposed tile is not
        // computed when 2 (tm / 2) + 1 < c / 128
        if (kSym && 2 * (tm >> 1) + 1 < (c >> 7)) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c + j < nh && r < pitch)
              __stcs(dist + (size_t)(c + j) * pitch + r,
                     (unsigned short)(r < nq ? acc[j] : (uint32_t)kKnnExcluded));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kGemmN));
  }
  if (threadIdx.x == 0 && failed)
    atomicOr(error, kGemmTimeout);
}

}  // namespace glp
