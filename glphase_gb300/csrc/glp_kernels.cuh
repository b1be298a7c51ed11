// glp_kernels.cuh -- sm_103a kernels for one MH generation of GLPhase's
// haplotype sampler: per-sample Metropolis-Hastings over surrogate-parent
// quadruples scored by the 4-state HMM forward likelihood, with the final
// haplotype sampling (hmm_work) fused into the same launch.
//
// Reference semantics (paths relative to the reference project root):
//   likelihood  Impute::hmm_like      src/impute.cpp:327-376 (CPU, float emit)
//               HMMLikeCUDA::hmmLike  src/hmmLike.cu:53-142  (GPU, VQ GLs)
//   MH chain    findHapSet            src/hmmLike.cu:145-217
//               Insti::solve          src/insti.cpp:1478-1551
//               MHSampler::SampleHap  src/MHSampler.hpp:81-96
//   sampling    Impute::hmm_work      src/impute.cpp:380-485
//
// Work decomposition (one warp = 32/P groups of P lanes, one sample per group):
//  * A sample's MH chain is inherently sequential, so its parallelism comes
//    from speculation: the P/2 lane pairs of a group evaluate the next P/2
//    evaluations of the chain (the current quadruple and the next proposals),
//    each built on the current state, i.e. assuming all earlier ones are
//    rejected.  The group then replays the accept rule in order; evaluations
//    after the first accepted proposal are discarded and re-evaluated from the
//    new state.  Decisions are exactly those of the sequential chain.
//  * A pair computes one likelihood: its even lane a forward pass over the
//    lower half of the sites, its odd lane a backward pass over the upper
//    half, both in one code path (x <- D T x), joined by a 4-term dot product
//    L = alpha_h . beta_h.  Half the sites per lane means half as many
//    speculative positions per round for the same lanes per sample, so fewer
//    of them are discarded.
//  * Scaling is by exact powers of two with an integer exponent per half;
//    the log-likelihood is assembled in binary64 (log(dot) + k*ln2).
//  * hmm_work runs one sample per thread in a second kernel over the final
//    quadruples, in the reference's exact binary32 operation order (no
//    contraction), so its output bits match the CPU reference.
//
// Memory (all resident in HBM across generations):
//   haps/hnew  uint64 [H][wn] hap-major   (parent words: L2-resident gathers)
//   emit       float4 [N][S]              (streamed, shared by a group)
//   packed     uint32 [ceil(S/8)][N]      (VQ codes; 16-entry table in smem)
//   tran4      float4 [S + 1]             (t0, t1, t2, t0 - t2); rows 0 and S = identity
//   tranp      float4 [S + 1]             (t1, t2, t0 - t2, t0 - t2), the pair rows the
//                                         blocked recursion stages (follows tran4)
//   beta       float4 [N][S]              (hmm_work scratch)
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "glp_join.h"
#include "glp_rng.h"
#include "glp_width.h"

namespace glp {

#ifndef GLP_GEN_WARPS
#define GLP_GEN_WARPS 4
#endif
constexpr int kWarps = GLP_GEN_WARPS;  // warps per generation block
constexpr int kThreads = 32 * kWarps;
// Most lanes per sample: teams of two and four warps are whole parts of a block.
constexpr uint32_t kWidest = kWarps % 4 == 0 ? 128 : kWarps % 2 == 0 ? 64 : 32;
// Resident blocks per SM the generation kernels are compiled for (the launch
// bound's minimum): with 3 the compiler may use up to 168 registers a thread and
// takes 120-136, so 3 blocks of the 8- and 16-lane kernels fit.  A bound of 4 (a cap
// of 128) was 2.4 % slower on 10,000 samples x 4,096 sites and 5 % on 2,000 x 8,192,
// 5 (a cap of 96) 16 %; of 2 the same.
#ifndef GLP_MIN_BLOCKS
#define GLP_MIN_BLOCKS 3
#endif
constexpr int kMinBlocks = GLP_MIN_BLOCKS;
constexpr uint32_t kNone = 0xffffffffu;
// Generation counters (GenParams::stats): scored evaluations, speculative
// rounds, accepted proposals, evaluations redone site by site after a block
// left the normalisation range, warp rounds, and active lanes summed over
// warp rounds.
constexpr int kStats = 6;
constexpr float kTiny = 0x1p-64f;
constexpr float kHuge = 0x1p64f;

struct GenParams {
  uint32_t N, S, C, H, wn, emit_mode;
  const uint64_t *__restrict__ haps;
  uint64_t *__restrict__ hnew;
  const float4 *__restrict__ emit;
  const float *__restrict__ prob;
  const float4 *__restrict__ tran4;
  const float4 *__restrict__ tranp;  // tran4's rows as (t1, t2, t0 - t2, t0 - t2)
  const uint32_t *__restrict__ packed;
  const float4 *__restrict__ vq_table;
  const uint32_t *__restrict__ quad_in;
  uint32_t *__restrict__ quad_out;
  const uint32_t *__restrict__ props;
  const uint8_t *__restrict__ tr_slot;
  const double *__restrict__ tr_u;
  const float *__restrict__ tr_work;
  double *__restrict__ like_out;
  double *__restrict__ eval_trace;
  uint8_t *__restrict__ accept_trace;
  float4 *__restrict__ beta;
  uint32_t *__restrict__ counter;
  unsigned long long *__restrict__ stats;
  int *__restrict__ error;
  const uint32_t *__restrict__ nbr;  // [N][klen] surrogate table, or null
  uint32_t klen, samp_lo, samp_hi;   // uniform surrogates over [samp_lo, samp_hi)
  uint32_t burnin;                   // >0: advance_kernel sets pen = min((g+1)/burnin,1)^2
  uint32_t kick;                     // 1: surrogates from [samp_lo, H) in generation 0 only
  uint32_t kick_first;               // 1: every chain's first proposal from the panel rows
  float pc[16];
  float pen;
  uint64_t seed;
  uint32_t generation;
  uint32_t do_work;
  uint32_t stream;  // 1: emission rows are asked for ahead (mark_stream)
  float rate;       // acceptance rate that a chain's speculation starts from
};

// ---------------------------------------------------------------------------
// Emission sources.  Both hand out the 4 emission values of a site,
// e[(father_bit << 1) | mother_bit] (impute.cpp:338-342).

// L1 prefetch of the line holding `ptr` (no register is held; the later
// load of the same line then hits L1).
__device__ __forceinline__ void prefetch_l1(const void *ptr) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(ptr));
}

// Bulk prefetch of [ptr, ptr + bytes) into L2 (a hint: nothing is written);
// ptr and bytes must be multiples of 16 and the range inside one allocation.
__device__ __forceinline__ void prefetch_l2_bulk(const void *ptr, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(ptr), "r"(bytes) : "memory");
}

// Asynchronous global -> shared copies (cp.async): the data lands in shared
// memory without occupying registers; cp_async_wait<n> returns once at most n
// of this thread's committed copy groups are still in flight.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int n>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(n));
}

// Staging of 8-site blocks: one slot = 8 transition rows followed by the 8
// sites' emission data (8 float4, or the block's VQ word in the first 4
// bytes).  A forward slot holds sites m0 .. m0+7 in order with the rows
// T_m0 .. T_m0+7 the forward recursion applies there; a backward slot holds
// sites n0+7 .. n0 (row j is site n0 + 7 - j) with the rows T_{n0+8-j} the
// backward recursion applies there, so both directions read slot row j at
// step j of a block.
constexpr int kSlotF4 = 16;
// Slots per direction: block t uses slot t mod 4, so within the 4-block
// quarter words the loop runs, every slot offset is a constant; two blocks
// are in flight while one is read.
constexpr int kRing = 4;
// A group's ring: forward slots at [0, 64) and backward slots at [68, 132)
// float4, so the forward and the backward row a group reads at one step are 4
// float4 (16 banks) apart; rings of neighbouring groups are 137 float4 apart
// (1 mod 8), so the 16-byte reads of the four 8-lane groups of a warp -- two
// rows a group -- fall in eight distinct bank quads.
constexpr int kBwdOffF4 = kRing * kSlotF4 + 4;
constexpr int kGroupF4 = kBwdOffF4 + kRing * kSlotF4;
constexpr int kGroupStrideF4 = kGroupF4 + 5;
static_assert(kGroupStrideF4 % 8 == 1 && kBwdOffF4 % 8 == 4, "ring bank layout");

// The rows of an 8-row block that lane li of a P-lane group copies: nr rows
// from rb.  From P = 8 up lanes 0..7 take one row each; narrower groups take
// 8/P consecutive rows per lane, so that one copy instruction of the warp
// writes rows 8/P apart in each group: with the groups' rings 1 mod 8 float4
// apart, the 16-byte writes of the groups in a quarter warp then fall in
// disjoint banks (consecutive rows per instruction would overlap).
struct StageRows {
  uint32_t rb, nr;
};
template <int kMaxRows>
__device__ __forceinline__ StageRows stage_rows(uint32_t li, uint32_t P) {
  StageRows r;
  if (kMaxRows == 1 || P >= 8) {  // kMaxRows == 1: the kernel's groups never narrow below 8
    r.rb = li;
    r.nr = li < 8 ? 1u : 0u;
  } else {
    r.nr = 8u >> (__ffs(P) - 1);  // 8 / P, P a power of two
    r.rb = li * r.nr;
  }
  return r;
}

// Copies 8 consecutive float4 from src into dst (stage8) or into dst in
// reverse order, dst[7 - i] = src[i] (stage8_rev): this lane's rows of the
// block (kMaxRows = 8/P bounds nr for the group size P the kernel starts
// with; a group only widens later).
template <int kMaxRows>
__device__ __forceinline__ void stage8(float4 *dst, const float4 *src, StageRows r) {
#pragma unroll
  for (uint32_t k = 0; k < (uint32_t)kMaxRows; ++k)
    if (k < r.nr)
      cp_async16(dst + r.rb + k, src + r.rb + k);
}
template <int kMaxRows>
__device__ __forceinline__ void stage8_rev(float4 *dst, const float4 *src, StageRows r) {
#pragma unroll
  for (uint32_t k = 0; k < (uint32_t)kMaxRows; ++k)
    if (k < r.nr)
      cp_async16(dst + 7 - (r.rb + k), src + r.rb + k);
}

// Emission sources.  stage / stage_rev copy one block's emission data into
// a forward / backward slot; block(src, rev) prepares a staged block and
// at(b, j) returns the emission of the slot's row j; get1(m) reads site m
// directly (the sites above the last full block, and the site-by-site pass).
struct EmitF32 {
  const float4 *row;
  using Blk = const float4 *;
  __device__ __forceinline__ void init(const GenParams &p, uint32_t s, const float4 *) {
    row = p.emit + (size_t)s * p.S;
  }
  __device__ __forceinline__ float4 get1(uint32_t m) const { return __ldg(row + m); }
  // asks L2 for the line of site m
  __device__ __forceinline__ void ahead(uint32_t m) const {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row + m));
  }
  // the sites m .. m + 3, m a multiple of 4, from global memory
  __device__ __forceinline__ void get4(uint32_t m, float4 (&e)[4]) const {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      e[j] = __ldg(row + m + j);
  }
  // copy block t (sites 8t .. 8t+7) into a forward / backward slot
  template <int kMaxRows>
  __device__ __forceinline__ void stage(float4 *dst, uint32_t t, StageRows r) const {
    stage8<kMaxRows>(dst, row + 8 * (size_t)t, r);
  }
  template <int kMaxRows>
  __device__ __forceinline__ void stage_rev(float4 *dst, uint32_t t, StageRows r) const {
    stage8_rev<kMaxRows>(dst, row + 8 * (size_t)t, r);
  }
  __device__ __forceinline__ Blk block(const float4 *src, bool) const { return src; }
  __device__ __forceinline__ float4 at(Blk b, uint32_t j) const { return b[j]; }
};

// 4-bit VQ codes, eight per uint32, most significant nibble first
// (glPack.cpp:104-109, hmmLike.cu:20-24), so one block of 8 sites is one
// word; table[c] = FillEmit(decode(c)) computed once on the host.  A backward
// slot holds the same word; block() reverses its nibbles so that code j is
// the site of row j.
struct EmitVQ {
  const uint32_t *col;
  const float4 *table;
  uint32_t stride;
  using Blk = uint32_t;
  __device__ __forceinline__ void init(const GenParams &p, uint32_t s, const float4 *tab) {
    col = p.packed + s;
    stride = p.N;
    table = tab;
  }
  __device__ __forceinline__ void ahead(uint32_t) const {}
  __device__ __forceinline__ void get4(uint32_t m, float4 (&e)[4]) const {
    const uint32_t w = __ldg(col + (size_t)(m >> 3) * stride) << (4u * (m & 4u));
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
      e[j] = table[(w >> (28u - 4u * j)) & 15u];
  }
  __device__ __forceinline__ float4 get1(uint32_t m) const {
    const uint32_t w = __ldg(col + (size_t)(m >> 3) * stride);
    return table[(w >> (28u - 4u * (m & 7u))) & 15u];
  }
  template <int kMaxRows>
  __device__ __forceinline__ void stage(float4 *dst, uint32_t t, StageRows r) const {
    if (r.rb == 0 && r.nr != 0)  // lane 0 of the group
      cp_async4(dst, col + (size_t)t * stride);
  }
  template <int kMaxRows>
  __device__ __forceinline__ void stage_rev(float4 *dst, uint32_t t, StageRows r) const {
    stage<kMaxRows>(dst, t, r);
  }
  __device__ __forceinline__ Blk block(const float4 *src, bool rev) const {
    const uint32_t w = *reinterpret_cast<const uint32_t *>(src);
    const uint32_t b = __byte_perm(w, 0u, 0x0123u);  // bytes reversed
    const uint32_t r = ((b >> 4) & 0x0f0f0f0fu) | ((b & 0x0f0f0f0fu) << 4);
    return rev ? r : w;
  }
  __device__ __forceinline__ float4 at(Blk w, uint32_t j) const {
    return table[(w >> (28u - 4u * j)) & 15u];
  }
};

// ---------------------------------------------------------------------------
// The 4-state recursion (impute.cpp:353-373).
//
// Both halves of an evaluation run in one form, x <- D_m (T x): the forward
// half carries alpha_m = D_m T_m alpha_{m-1} up from site 0 (T_0 = I on the
// uniform start); the backward half carries v_m = D_m beta_m = D_m T_{m+1}
// v_{m+1} down from the top site (T_S = I on the all-ones start).  The two
// meet at L = alpha_h . (T_{h+1} v_{h+1}).  T is symmetric, so this is the
// reference's likelihood; one code path serves both halves.

// The state in register pairs for the packed binary32 instructions of
// sm_100+ (__ffma2_rn and friends round each component as the scalar
// instruction does): X = (l00, l01), Y = (l11, l10), P = (p2, p1) with
// p1 = l01 + l10 and p2 = l00 + l11, so that X + Y = P.
struct FState {
  float2 X, Y, P;
  int k;
};

__device__ __forceinline__ void fstate_fill(FState &f, float l, int k) {
  f.X = f.Y = make_float2(l, l);
  f.P = make_float2(l + l, l + l);
  f.k = k;
}

__device__ __forceinline__ void select4(const float4 e, bool a0, bool a1, bool c0,
                                        bool c1, float &s00, float &s01, float &s10,
                                        float &s11) {
  const float lo0 = a0 ? e.z : e.x, hi0 = a0 ? e.w : e.y;
  const float lo1 = a1 ? e.z : e.x, hi1 = a1 ? e.w : e.y;
  s00 = c0 ? hi0 : lo0;
  s01 = c1 ? hi0 : lo0;
  s10 = c0 ? hi1 : lo1;
  s11 = c1 ? hi1 : lo1;
}

__device__ __forceinline__ void fstate_scale(FState &f, float sc) {
  const float2 s2 = make_float2(sc, sc);
  f.X = __fmul2_rn(f.X, s2);
  f.Y = __fmul2_rn(f.Y, s2);
  f.P = __fmul2_rn(f.P, s2);
}

// One step with per-site power-of-two rescaling (the site-by-site pass), for
// t = (x, y, z, x - z).
__device__ __forceinline__ void fwd_step(FState &f, const float4 t, float s00, float s01,
                                         float s10, float s11) {
  const float l00 = f.X.x, l01 = f.X.y, l10 = f.Y.y, l11 = f.Y.x, p1 = f.P.y, p2 = f.P.x;
  const float b00 = fmaf(l11, t.z, fmaf(p1, t.y, l00 * t.x));
  const float b01 = fmaf(l10, t.z, fmaf(p2, t.y, l01 * t.x));
  const float b10 = fmaf(l01, t.z, fmaf(p2, t.y, l10 * t.x));
  const float b11 = fmaf(l00, t.z, fmaf(p1, t.y, l11 * t.x));
  f.X = make_float2(b00 * s00, b01 * s01);
  f.Y = make_float2(b11 * s11, b10 * s10);
  f.P = __fadd2_rn(f.X, f.Y);
  if (f.P.x + f.P.y < kTiny) {
    fstate_scale(f, kHuge);
    f.k -= 64;
  }
}

// fwd_step's products and sums in its order, two at a time, without its
// rescaling; returns the state's sum.
__device__ __forceinline__ float fwd_step_free(FState &f, const float4 t, float2 sx, float2 sy) {
  const float2 tx = make_float2(t.x, t.x), ty = make_float2(t.y, t.y),
               tz = make_float2(t.z, t.z), c = make_float2(f.P.y, f.P.x);
  const float2 bx = __ffma2_rn(f.Y, tz, __ffma2_rn(c, ty, __fmul2_rn(f.X, tx)));
  const float2 by = __ffma2_rn(f.X, tz, __ffma2_rn(c, ty, __fmul2_rn(f.Y, tx)));
  f.X = __fmul2_rn(bx, sx);
  f.Y = __fmul2_rn(by, sy);
  f.P = __fadd2_rn(f.X, f.Y);
  return f.P.x + f.P.y;
}

// The same step without rescaling, in a shared-term form of T: with
// p1 = l01 + l10 and p2 = l00 + l11,
//   (T l)_00 = (x - z) l00 + c1,  (T l)_11 = (x - z) l11 + c1,  c1 = y p1 + z p2
//   (T l)_01 = (x - z) l01 + c2,  (T l)_10 = (x - z) l10 + c2,  c2 = y p2 + z p1
// so that X <- (w X + c) * sx and Y <- (w Y + c) * sy for c = (c1, c2),
// w = x - z: four scalar and five packed instructions a site.  t is a row of
// the pair table, (y, z, w, w), whose last two components form the pair
// (w, w).  The caller keeps the state in range by normalising at block
// boundaries.
__device__ __forceinline__ void fwd_fast(FState &f, const float4 t, float2 sx, float2 sy) {
  const float2 c = make_float2(fmaf(t.y, f.P.x, t.x * f.P.y), fmaf(t.y, f.P.y, t.x * f.P.x));
  const float2 w = make_float2(t.z, t.w);
  f.X = __fmul2_rn(__ffma2_rn(w, f.X, c), sx);
  f.Y = __fmul2_rn(__ffma2_rn(w, f.Y, c), sy);
  f.P = __fadd2_rn(f.X, f.Y);
}

// x <- T x alone (the backward half's last step, T_{h+1} v_{h+1}), for
// t = (x, y, z, x - z).
__device__ __forceinline__ void apply_tran(FState &f, const float4 t) {
  const float2 c = make_float2(fmaf(t.z, f.P.x, t.y * f.P.y), fmaf(t.z, f.P.y, t.y * f.P.x));
  const float2 w = make_float2(t.w, t.w);
  f.X = __ffma2_rn(w, f.X, c);
  f.Y = __ffma2_rn(w, f.Y, c);
}

// Exact power-of-two normalisation at a block boundary: scales the state so
// that its sum lies in [2^62, 2^63).  Starting a block of 8 sites in that
// range, the sums stay normal floats as long as the block shrinks them by less
// than 2^-124 (emissions are at most 1, so sums never grow).  The return
// value is e - 65 for the sum's biased exponent e: it lies outside [0, 127]
// exactly when the sum left [2^-62, 2^66), i.e. when range may have been lost
// in the block just computed (the scale is then meaningless too) and the
// evaluation must be redone with per-site rescaling.
__device__ __forceinline__ uint32_t fwd_norm(FState &f) {
  const uint32_t eb = __float_as_uint(f.P.x + f.P.y) & 0x7f800000u;
  fstate_scale(f, __uint_as_float(0x9e000000u - eb));  // 2^(189 - e)
  const int e = (int)(eb >> 23);
  f.k += e - 189;
  return (uint32_t)(e - 65);
}
// The same for a state kept in range site by site (any sum down to 2^-65 is
// legitimate there): the exponent is clamped so the scale stays a normal float.
__device__ __forceinline__ void fwd_renorm(FState &f) {
  const int e = (int)((__float_as_uint(f.P.x + f.P.y) >> 23) & 0xffu);
  const int ec = max(e, 62);
  fstate_scale(f, __uint_as_float((uint32_t)(316 - ec) << 23));  // 2^(189 - ec)
  f.k += ec - 189;
}

// Overflow guard of the site-by-site pass (emissions above 1 could grow it).
__device__ __forceinline__ void fwd_guard(FState &f) {
  if (f.P.x + f.P.y > kHuge) {
    fstate_scale(f, kTiny);
    f.k += 64;
  }
}

struct Parents {
  uint64_t f0, f1, m0, m1;
};

__device__ __forceinline__ Parents load_parents(const uint64_t *haps, uint32_t wn, uint4 q,
                                                uint32_t w) {
  Parents r;
  r.f0 = __ldg(haps + (size_t)q.x * wn + w);
  r.f1 = __ldg(haps + (size_t)q.y * wn + w);
  r.m0 = __ldg(haps + (size_t)q.z * wn + w);
  r.m1 = __ldg(haps + (size_t)q.w * wn + w);
  return r;
}

// Bit-reversed parent words: bit 63 - i holds site i of the word, so the
// backward half reads its descending sites as ascending bits.
__device__ __forceinline__ Parents reverse_parents(const Parents &p) {
  Parents r;
  r.f0 = __brevll(p.f0);
  r.f1 = __brevll(p.f1);
  r.m0 = __brevll(p.m0);
  r.m1 = __brevll(p.m1);
  return r;
}

__device__ __forceinline__ void prefetch_parents(const uint64_t *haps, uint32_t wn, uint4 q,
                                                 uint32_t w) {
  prefetch_l1(haps + (size_t)q.x * wn + w);
  prefetch_l1(haps + (size_t)q.y * wn + w);
  prefetch_l1(haps + (size_t)q.z * wn + w);
  prefetch_l1(haps + (size_t)q.w * wn + w);
}

// 32-bit halves of the four parent words: the bits of four 8-site blocks.
struct Bits32 {
  uint32_t f0, f1, m0, m1;
};

__device__ __forceinline__ Bits32 half_words(const Parents &pw, uint32_t h) {
  Bits32 r;
  r.f0 = (uint32_t)(pw.f0 >> (32 * h));
  r.f1 = (uint32_t)(pw.f1 >> (32 * h));
  r.m0 = (uint32_t)(pw.m0 >> (32 * h));
  r.m1 = (uint32_t)(pw.m1 >> (32 * h));
  return r;
}

// The emissions of one site as the pairs (s00, s01) and (s11, s10) that
// multiply X and Y.
__device__ __forceinline__ void site_emission(const float4 e, const Bits32 &bw, uint32_t j,
                                              float2 &sx, float2 &sy) {
  const uint32_t bit = 1u << j;  // j is a compile-time constant in the unrolled block
  select4(e, (bw.f0 & bit) != 0u, (bw.f1 & bit) != 0u, (bw.m0 & bit) != 0u,
          (bw.m1 & bit) != 0u, sx.x, sx.y, sy.y, sy.x);
}

// One staged block of 8 sites: row j of the slot (transition rows first,
// emission data from slot + 8) with bit 8B + j of the parent halves; the
// state is normalised at the end (kSub = 2: also after the first 4 sites)
// and eacc collects the range codes.
template <int B, class E, int kSub>
__device__ __forceinline__ void block8(FState &x, const E &em, const float4 *slot,
                                       typename E::Blk eb, const Bits32 &bw, uint32_t &eacc) {
#pragma unroll
  for (uint32_t j = 0; j < 8; ++j) {
    const float4 e = em.at(eb, j), t = slot[j];
    float2 sx, sy;
    site_emission(e, bw, 8 * B + j, sx, sy);
    fwd_fast(x, t, sx, sy);
    if (kSub == 2 && j == 3)
      eacc |= fwd_norm(x);
  }
  eacc |= fwd_norm(x);
}

// Log-likelihood of one quadruple by a plain forward pass, site by site, with
// the per-site power-of-two rescaling of fwd_step (the scheme of
// impute.cpp:327-376), reading emission, transition and parent words straight
// from global memory, four sites' rows at a time.  Used, rarely, for an evaluation
// whose blocked pass may have lost range: a lone lane's walk, so that a generation
// ends as late as its redos follow one another (400 x 2,048 with every evaluation made
// again 4.10 ms, from codes 5.01; with one site's rows at a time 5.81 and 8.38).
template <class E>
__device__ __noinline__ double like_forward(const uint64_t *__restrict__ haps, uint32_t wn,
                                            uint32_t S, const float4 *__restrict__ tran4,
                                            const E em, uint4 q) {
  FState f;
  fstate_fill(f, 0.25f, 0);
  for (uint32_t w = 0; w < wn; ++w) {
    const Parents pw = load_parents(haps, wn, q, w);
    const uint32_t end = min(S, (w + 1) * 64);
    auto site = [&](const float4 e, const float4 t, uint32_t j) {
      float s00, s01, s10, s11;
      select4(e, (pw.f0 >> j) & 1, (pw.f1 >> j) & 1, (pw.m0 >> j) & 1, (pw.m1 >> j) & 1, s00,
              s01, s10, s11);
      fwd_step(f, t, s00, s01, s10, s11);
    };
    uint32_t m = w * 64;
#pragma unroll 1
    for (; m + 4 <= end; m += 4) {  // four sites' rows loaded together
      float4 e[4], t[4];
      em.get4(m, e);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        t[j] = __ldg(tran4 + m + j);
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
        site(e[j], t[j], (m & 63u) + j);
    }
#pragma unroll 1
    for (; m < end; ++m)
      site(em.get1(m), __ldg(tran4 + m), m & 63u);
    fwd_guard(f);
  }
  const double sum = (((double)f.X.x + (double)f.X.y) + (double)f.Y.y) + (double)f.Y.x;
  return log(sum) + (double)f.k * 0.69314718055994530942;
}

// ln(x . y) + k ln 2 over the four states, in natural log and binary64.  The
// exponent of the product joins k exactly, and the logarithm of its mantissa in
// [1, 2) is taken in binary32 (absolute error below 3e-7, against
// log-likelihoods of order -S), so binary64 only adds the two parts: its pipe
// takes an instruction of a warp in 16 cycles.  For the same reason the mantissa
// comes from pairs of floats where those give the same float as the binary64
// product, and else from that (glp_join.h).  In binary64 alone the products, sums
// and conversions took 820 cycles of a round that has 3,600 beside its sites, as
// pairs 70; the test for the other case adds 0.1 us a round (a generation of 3 x 3
// sites 83.4 and 84.5 us, larger ones within 0.2 %).
__device__ __forceinline__ double log_dot(float2 xX, float2 xY, float2 yX, float2 yY, int k) {
  constexpr double kLn2 = 0.69314718055994530942;
  float m;
  int e;
  if (!join_product(xX.x, xX.y, xY.y, xY.x, yX.x, yX.y, yY.y, yY.x, m, e)) {
    const double dot = (double)xX.x * (double)yX.x + (double)xX.y * (double)yX.y +
                       (double)xY.y * (double)yY.y + (double)xY.x * (double)yY.x;
    if (!(dot > 0x1p-1000))
      return log(dot) + (double)k * kLn2;
    const long long bits = __double_as_longlong(dot);
    e = (int)((bits >> 52) & 0x7ff) - 1023;
    m = (float)__longlong_as_double((bits & 0x000fffffffffffffLL) | 0x3ff0000000000000LL);
  }
  return (double)logf(m) + (double)(e + k) * kLn2;
}

// Log-likelihood (natural log, binary64) of quadruple q, scored by a lane
// pair of a P-lane group.  Of the nw = floor(S/64) full 64-site words, the
// even lane runs the forward half over words [0, wf), wf = ceil(nw/2); the
// odd lane first runs the sites of the partial top word (straight from
// global memory), then the backward half over words
// [wf, nw) from the top.  Each word is eight 8-site blocks, run four at a
// time so that ring slots and parent-bit positions are constants: step t
// stages forward block t and backward block 8 nw - 1 - t of every pair into
// the group's ring (cp.async, two steps ahead), so the arithmetic reads
// shared memory only.  With an odd word count the odd lane idles through
// the last word (it computes on stale rows and restores its state after).
// States are normalised at block boundaries (exact powers of two); a
// quadruple whose block sums left the safe range is recomputed site by site
// by the even lane.  The pair joins with two exact-product shuffles, so both
// lanes return the same value.  All P lanes of the group call this together;
// gmask names the lanes that synchronise at each step (the group, or the
// whole warp when every group runs the same loop).  tran4 and tranp hold
// S + 1 rows, rows 0 and S the identity; the ring stages tranp's.
// kFull: every lane of the warp takes part (gmask is the full mask, known to
// the compiler).
template <int kMaxRows, class E, int kSub = 1, bool kFull = false, bool kAhead = false>
__device__ __forceinline__ double eval_pair(const GenParams &p, const E &em, uint4 q,
                                            float4 *stage, uint32_t li, uint32_t P,
                                            unsigned gmask_in) {
  const unsigned gmask = kFull ? 0xffffffffu : gmask_in;
  const uint32_t S = p.S, wn = p.wn;
  const float4 *tran4 = p.tran4, *tranp = p.tranp;
  const bool bwd = (li & 1u) != 0;
  const uint32_t nw = S >> 6, wf = (nw + 1) >> 1, wb = nw - wf;
  const uint32_t nbf = 8 * wf, nbb = 8 * wb, top = 8 * nw - 1;  // blocks per direction
  // block-normalised states start at sum 2^62: the forward state 1/4 scaled
  // by 2^62, the backward state 1 scaled by 2^60
  FState x;
  fstate_fill(x, 0x1p60f, bwd ? -60 : -62);
  uint32_t eacc = 0;  // OR of the blocks' range codes (fwd_norm)
  float4 *const stF = stage, *const stB = stage + kBwdOffF4;
  const StageRows rows = stage_rows<kMaxRows>(li, P);
  // block t0 + d of both directions into slot (t0 + d) mod 4: forward sites
  // 8t .. 8t+7 with rows T_8t .., backward sites of block top - t reversed
  // with the rows T_{m+1} of its sites m.  t0 is a multiple of 4 and d a
  // constant, so the sources are base pointers of the quarter word plus
  // constant offsets.
  auto issue = [&](uint32_t t0, uint32_t d) {
    const uint32_t t = t0 + d, slot = d & 3u;
    if (t < nbf) {
      stage8<kMaxRows>(stF + slot * kSlotF4, tranp + 8 * (size_t)t0 + 8 * d, rows);
      em.template stage<kMaxRows>(stF + slot * kSlotF4 + 8, t, rows);
    }
    if (t < nbb) {
      stage8_rev<kMaxRows>(stB + slot * kSlotF4, tranp + 8 * (size_t)(top - t0) + 1 - 8 * d,
                           rows);
      em.template stage_rev<kMaxRows>(stB + slot * kSlotF4 + 8, top - t, rows);
    }
    cp_async_commit();
  };
  issue(0, 0);
  issue(0, 1);
  if (bwd && (S & 63u)) {
    // the sites of the partial top word: four at a time, their rows loaded
    // together and the test for the rescaling of fwd_step made once for the four;
    // where it would have rescaled, and for the sites above the last whole four,
    // site by site.  A lone warp takes 83 cycles a site, and 49 in a whole word
    // (site by site 120; a generation of 60 x 1,000 0.654 and 0.617 ms).  Two
    // fours in registers at once were slower: 168 registers, with spills.
    const Parents pw = load_parents(p.haps, wn, q, nw);
#pragma unroll 1
    for (int lo = (int)((S - 1) & ~3u), n = (int)S - lo; lo >= (int)(nw * 64); lo -= 4, n = 4) {
      const uint32_t sh = (uint32_t)lo & 63u;
      float low = 0.0f;
      FState y = x;
      if (n == 4) {
        const Bits32 bw = {(uint32_t)(pw.f0 >> sh), (uint32_t)(pw.f1 >> sh),
                           (uint32_t)(pw.m0 >> sh), (uint32_t)(pw.m1 >> sh)};
        float4 e[4], t[4];
        em.get4((uint32_t)lo, e);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          t[j] = __ldg(tran4 + lo + 1 + j);
        low = kHuge;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          float2 sx, sy;
          site_emission(e[j], bw, j, sx, sy);
          low = fminf(low, fwd_step_free(y, t[j], sx, sy));
        }
      }
      if (low >= kTiny) {
        x = y;
      } else {
#pragma unroll 1
        for (int j = n - 1; j >= 0; --j) {
          const uint32_t i = sh + (uint32_t)j;
          float s00, s01, s10, s11;
          select4(em.get1((uint32_t)(lo + j)), (pw.f0 >> i) & 1, (pw.f1 >> i) & 1,
                  (pw.m0 >> i) & 1, (pw.m1 >> i) & 1, s00, s01, s10, s11);
          fwd_step(x, __ldg(tran4 + lo + j + 1), s00, s01, s10, s11);
        }
      }
    }
    fwd_renorm(x);
  }
  float4 *const mine = bwd ? stB : stF;
#pragma unroll 1
  for (uint32_t i = 0; i < wf; ++i) {
    const bool act = !bwd || i < wb;
    const FState xs = x;
    const uint32_t es = eacc;
    const uint32_t w = bwd ? nw - 1 - i : i;
    const Parents raw = load_parents(p.haps, wn, q, w);
    const Parents pw = bwd ? reverse_parents(raw) : raw;
    if (i + 1 < (bwd ? wb : wf))  // this lane's next word
      prefetch_parents(p.haps, wn, q, bwd ? w - 1 : w + 1);
    // Rows that come from memory each round are asked for a word (1 KB a
    // direction) ahead where few warps hide the latency: two staged blocks are
    // less than it (2,000 x 8,192 at 8 lanes: 5.19 and 4.46 ms; at 16 lanes no
    // change, and for rows in L2 1.5 % slower).
    if (kMaxRows > 1 || kAhead) {
      if (p.stream)
        for (uint32_t l = li; l < 8; l += P) {
          if (i + 1 < wf)
            em.ahead(64 * (i + 1) + 8 * l);
          if (i + 1 < wb)
            em.ahead(64 * (nw - 2 - i) + 8 * l);
        }
    }
#pragma unroll 1
    for (uint32_t h = 0; h < 2; ++h) {
      const uint32_t t0 = 8 * i + 4 * h;
      const Bits32 bw = half_words(pw, h);
#pragma unroll
      for (uint32_t b = 0; b < 4; ++b) {
        // One barrier a block: the slot staged here, (t + 2) mod 4, was last
        // read at step t - 2, which every lane of the group finished before
        // the barrier of step t - 1 let this one go on.
        issue(t0, b + 2);
        cp_async_wait<2>();
        __syncwarp(gmask);
        const float4 *slot = mine + b * kSlotF4;
        switch (b) {  // bit positions 8b + j as constants
          case 0: block8<0, E, kSub>(x, em, slot, em.block(slot + 8, bwd), bw, eacc); break;
          case 1: block8<1, E, kSub>(x, em, slot, em.block(slot + 8, bwd), bw, eacc); break;
          case 2: block8<2, E, kSub>(x, em, slot, em.block(slot + 8, bwd), bw, eacc); break;
          default: block8<3, E, kSub>(x, em, slot, em.block(slot + 8, bwd), bw, eacc); break;
        }
      }
    }
    if (!act) {  // the odd lane's idle word
      x = xs;
      eacc = es;
    }
  }
  if (bwd)  // beta_{64 wf - 1} = T_{64 wf} v_{64 wf} (row S is the identity)
    apply_tran(x, __ldg(tran4 + 64 * (size_t)wf));
  // alpha . beta on both lanes: the same products, and sums of the same pairs
  const float2 yX = make_float2(__shfl_xor_sync(gmask, x.X.x, 1),
                                __shfl_xor_sync(gmask, x.X.y, 1)),
               yY = make_float2(__shfl_xor_sync(gmask, x.Y.x, 1),
                                __shfl_xor_sync(gmask, x.Y.y, 1));
  const int yk = __shfl_xor_sync(gmask, x.k, 1);
  const uint32_t bad = (eacc | __shfl_xor_sync(gmask, eacc, 1)) & ~127u;
  double L = log_dot(x.X, x.Y, yX, yY, x.k + yk);
  if (__any_sync(gmask, bad != 0u)) {
    double Lf = L;
    if (bad && !bwd) {
      if (p.stats)
        atomicAdd(p.stats + 3, 1ull);
      Lf = like_forward(p.haps, wn, S, tran4, em, q);
    }
    L = __shfl_sync(gmask, Lf, (threadIdx.x & 31u) & ~1u);
  }
  return L;
}

// ---------------------------------------------------------------------------
// hmm_work, binary32 in the reference's operation order
// (impute.cpp:380-485): explicit _rn intrinsics keep nvcc from contracting
// products and sums into FMAs, so results are bit-identical to the CPU code.

__device__ __forceinline__ float fma3_rn(float a0, float b0, float a1, float b1, float a2,
                                         float b2, float a3, float b3) {
  // ((a0*b0 + a1*b1) + a2*b2) + a3*b3, every product and sum rounded.
  return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a0, b0), __fmul_rn(a1, b1)),
                             __fmul_rn(a2, b2)),
                   __fmul_rn(a3, b3));
}

// hmm_work is split in two passes with the reference's arithmetic unchanged.
// The forward state l_m of impute.cpp:416-447 does not depend on the sampled
// bits, so (1) the two sequential recursions -- the backward vectors beta_m
// (impute.cpp:389-414) and the forward l_m -- run per sample and leave
// p_m = l_m * beta_m (the products of impute.cpp:449-452) in the scratch;
// (2) the sampling of impute.cpp:453-484 then runs for every site in parallel,
// one warp per part of a sample and 32 sites per instruction.
//
// Pass 1: a block of two warps takes 32 samples of one chunk, one lane a
// sample.  Warp 0 runs the backward recursion from the top site, warp 1 the
// forward recursion from site 0, at the same time.  Neither depends on the other
// until p, so each runs to the middle storing its vectors; after a block barrier
// each goes on through the other half, where it multiplies its vectors with the
// stored ones.
//
// What bounds it: with a recursion warp a scheduler or less, the instructions
// that a step issues, each about two cycles apart (a step's dependent chain, 16
// instructions and a reciprocal, is shorter); with more, the 80 bytes a site and
// sample that it moves (at 10,000 samples 4.2 TB/s).  So the four states sit in
// one lane as two register pairs (shared between two lanes, every step waits for
// a shuffle) whose products are packed binary32 instructions, the reciprocal is a
// Newton step without a range test, and rows come (cp.async) and vectors go a
// tile of 8 sites at a time, 8 lanes a row.  Pass 1 before (a lane pair a
// recursion, blocks of 16 samples) and now: 256 x 1,024 0.156 and 0.099 ms, 2,000
// x 8,192 1.19 and 0.81, 10,000 x 4,096 1.16 and 0.80.  Measured and not kept:
// warps that pick the emissions and store the vectors beside each recursion warp
// (0.084 ms at 256 x 1,024, but 1.02 at 10,000 x 4,096: a barrier a tile couples
// them to the slowest), and the vectors of a half recomputed from states at the
// tiles' starts with the sampling in the same kernel (48 bytes a site instead of
// 108 for both passes, but ten warps in step: 0.127 against 0.117 ms for both
// passes and 1.2 against 1.05).
constexpr int kChainTile = 8;           // sites
constexpr int kChainRing = 4;           // tiles: one read, one next, two in flight
constexpr uint32_t kChainSamples = 32;  // samples per block
// A tile in shared memory keeps a sample's sites together, as in global memory
// (a copy of 8 lanes lands as one 128-byte write; sites apart, it took eight),
// rows 9 float4 apart: 1 mod 8, so that 8 samples' reads of a site fall in 8 quads.
constexpr uint32_t kRowF4 = kChainTile + 1;
constexpr uint32_t kTileF4 = kChainSamples * kRowF4;
constexpr int kChainThreads = 64;

// A vector over the four states, as the pairs (00, 01) and (11, 10): packed
// binary32 products then round each component as the scalar ones do.
struct States {
  float2 P, Q;
};
__device__ __forceinline__ States states_of(const float4 v) {
  return States{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float4 f4_of(const States v) {
  return make_float4(v.P.x, v.P.y, v.Q.x, v.Q.y);
}
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }
// The sums of two pairs as scalar additions: a packed addition of a packed
// product is contracted to a fused multiply-add, which rounds once.
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
  return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}

struct ChainTiles {  // of one recursion
  float4 e[kChainRing][kTileF4];  // emission rows
  float4 v[kChainRing][kTileF4];  // vectors: the stored ones in, the new ones out
  float4 t[kChainRing][kChainTile];  // transition rows
};

// 1 / x correctly rounded, for x in [2^-126, 2^126]: one Newton step y + y (1 - x y),
// each product and sum fused, from the approximate reciprocal y.  Where y is within
// a unit of its last place, 1 - x y is exact and the step's result correctly rounded
// but for a mantissa of ones (P. Markstein, IA-64 and Elementary Functions, 2000,
// chapter 8); that it is for every x of the range, those too, is what
// test_gpu_reciprocal.py compares, float by float.  Outside: NaN below, 0 above, NaN
// for infinity.
__device__ __forceinline__ float recip_newton(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}

// The same for any x: below 2^-126 by way of x 2^64 (both scalings are exact, or
// overflow as the reciprocal does), 0 and above 2^126 by __frcp_rn.
__device__ __forceinline__ float recip_any(float x) {
  const float a = fabsf(x), scale = a < 0x1p-126f ? 0x1p64f : 1.0f;
  const float r = recip_newton(x * scale) * scale;
  return a == 0.0f || a > 0x1p126f ? __frcp_rn(x) : r;
}

// The normalisation of a step (impute.cpp:404-409, 441-446): the sum in the
// reference's order, its reciprocal (kSafe: for any sum) and the four products.
// seen turns NaN with the reciprocal.
template <bool kSafe>
__device__ __forceinline__ States work_normalise(const States n, float &seen) {
  const float sum = __fadd_rn(__fadd_rn(__fadd_rn(n.P.x, n.P.y), n.Q.y), n.Q.x);
  const float inv = kSafe ? recip_any(sum) : recip_newton(sum);
  seen = fmaf(inv, 0.0f, seen);
  return States{__fmul2_rn(n.P, dup2(inv)), __fmul2_rn(n.Q, dup2(inv))};
}

// One step of the backward recursion from beta_m to beta_{m-1}
// (impute.cpp:389-414): emissions s and transition row t of site m.
template <bool kSafe>
__device__ __forceinline__ States work_bwd_step(const States v, const States s, const float4 t,
                                                float &seen) {
  const float2 P = __fmul2_rn(v.P, s.P), Q = __fmul2_rn(v.Q, s.Q);
  // (b01 + b10, b00 + b11) y
  const float2 c = __fmul2_rn(make_float2(__fadd_rn(P.y, Q.y), __fadd_rn(P.x, Q.x)),
                              dup2(t.y));
  const float2 x = dup2(t.x), z = dup2(t.z);
  return work_normalise<kSafe>(
      States{add_pair(add_pair(__fmul2_rn(P, x), c), __fmul2_rn(Q, z)),
             add_pair(add_pair(__fmul2_rn(Q, x), c), __fmul2_rn(P, z))},
      seen);
}

// One step of the forward recursion from l_{m-1} to l_m (impute.cpp:416-447):
// emissions s and transition row t of site m.  Site 0's row is the identity, so
// from the uniform 1/4 its step is the reference's first one, l = e / 4.
template <bool kSafe>
__device__ __forceinline__ States work_fwd_step(const States v, const States s, const float4 t,
                                                float &seen) {
  const float2 xy = make_float2(t.x, t.y), yx = make_float2(t.y, t.x), yz = make_float2(t.y, t.z),
               zy = make_float2(t.z, t.y);
  const float2 l00 = dup2(v.P.x), l01 = dup2(v.P.y), l10 = dup2(v.Q.y), l11 = dup2(v.Q.x);
  // ((l00 . + l01 .) + l10 .) + l11 . for (00, 01) and for (11, 10)
  const float2 P = add_pair(add_pair(add_pair(__fmul2_rn(l00, xy), __fmul2_rn(l01, yx)),
                                         __fmul2_rn(l10, yz)),
                              __fmul2_rn(l11, zy));
  const float2 Q = add_pair(add_pair(add_pair(__fmul2_rn(l00, zy), __fmul2_rn(l01, yz)),
                                         __fmul2_rn(l10, yx)),
                              __fmul2_rn(l11, xy));
  return work_normalise<kSafe>(States{__fmul2_rn(P, s.P), __fmul2_rn(Q, s.Q)}, seen);
}

__device__ __forceinline__ States mul_states(const States a, const States b) {
  return States{__fmul2_rn(a.P, b.P), __fmul2_rn(a.Q, b.Q)};
}

// The emissions of a site for the parents' bits a0, a1 (father), c0, c1 (mother).
__device__ __forceinline__ States pick_states(const float4 e, bool a0, bool a1, bool c0, bool c1) {
  States s;
  select4(e, a0, a1, c0, c1, s.P.x, s.P.y, s.Q.y, s.Q.x);
  return s;
}

__device__ __forceinline__ void cp_async16_cg(void *smem, const void *gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// One recursion over n tiles from state v: ascending from base0 (kFwd) or
// descending.  kComb: the other recursion's vectors are staged with the
// emissions and the products p are stored; else the vectors are.  Lane l has
// sample s0 + l with the final quadruple q (lanes past the chunk's end repeat its
// last sample and store nothing).  kSafe: reciprocals for any sum.
template <bool kFwd, bool kComb, bool kSafe>
__device__ __forceinline__ void chain_run(const GenParams &p, ChainTiles &sm, uint32_t lane,
                                          uint32_t s0, uint4 q, States &v, float &seen, int base0,
                                          int n) {
  if (n <= 0)
    return;
  const uint32_t S = p.S, unit = lane & 7u, r0 = lane >> 3;  // staging: 8 lanes a row
  const uint32_t last = min(kChainSamples, p.N - s0) - 1;  // rows past it repeat it
  const float4 *const emit = p.emit + (size_t)s0 * S;
  float4 *const beta = p.beta + (size_t)s0 * S;
  auto base_of = [&](int k) { return kFwd ? base0 + kChainTile * k : base0 - kChainTile * k; };
  auto stage = [&](int k) {
    if (k < n) {
      const uint32_t b = (uint32_t)base_of(k), m = min(b + unit, S - 1u);
      const int slot = k & (kChainRing - 1);
#pragma unroll
      for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t at = (r0 + 4 * i) * kRowF4 + unit;
        const size_t from = (size_t)min(r0 + 4 * i, last) * S + m;
        cp_async16_cg(&sm.e[slot][at], emit + from);
        if (kComb)
          cp_async16_cg(&sm.v[slot][at], beta + from);
      }
      if (lane < (uint32_t)kChainTile)
        cp_async16(&sm.t[slot][lane], p.tran4 + m);
    }
    cp_async_commit();
  };
  // the rows of four sites of a tile, in step order
  struct Rows {
    float4 e[4], t[4], o[4];
  };
  auto load = [&](Rows &r, int k, int half) {
    const int slot = k & (kChainRing - 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = 4 * half + j, o = kFwd ? i : kChainTile - 1 - i;
      r.e[j] = sm.e[slot][lane * kRowF4 + o];
      r.t[j] = sm.t[slot][o];
      if (kComb)
        r.o[j] = sm.v[slot][lane * kRowF4 + o];
    }
  };
  int w = base0 >> 6;
  const int w_end = base_of(n - 1) >> 6, dir = kFwd ? 1 : -1;
  Parents cur = load_parents(p.haps, p.wn, q, (uint32_t)w), next = cur;
  if (w != w_end)
    next = load_parents(p.haps, p.wn, q, (uint32_t)(w + dir));
  stage(0);
  stage(1);
  cp_async_wait<1>();
  __syncwarp();
  Rows ra, rb;
  load(ra, 0, 0);
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const int slot = k & (kChainRing - 1), base = base_of(k);
    stage(k + 2);  // the slot's last tile was stored two tiles ago
    if ((base >> 6) != w) {
      w = base >> 6;
      cur = next;
      if (w != w_end)
        next = load_parents(p.haps, p.wn, q, (uint32_t)(w + dir));
    }
    const int sh = base & 63;
    const uint32_t A0 = (uint32_t)(cur.f0 >> sh), A1 = (uint32_t)(cur.f1 >> sh),
                   C0 = (uint32_t)(cur.m0 >> sh), C1 = (uint32_t)(cur.m1 >> sh);
    float4 *const out = &sm.v[slot][lane * kRowF4];
    auto step = [&](int o, const float4 e, const float4 t, const float4 other) {
      const uint32_t bit = 1u << o;
      const States s = pick_states(e, A0 & bit, A1 & bit, C0 & bit, C1 & bit);
      if (kFwd)
        v = work_fwd_step<kSafe>(v, s, t, seen);
      out[o] = f4_of(kComb ? mul_states(v, states_of(other)) : v);
      if (!kFwd)
        v = work_bwd_step<kSafe>(v, s, t, seen);
    };
    auto four = [&](const Rows &r, int half) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = 4 * half + j;
        step(kFwd ? i : kChainTile - 1 - i, r.e[j], r.t[j], r.o[j]);
      }
    };
    const bool whole = base + kChainTile <= (int)S;
    if (whole) {
      load(rb, k, 1);
      four(ra, 0);
    }
    cp_async_wait<1>();
    __syncwarp();  // tile k + 1 has arrived
    if (k + 1 < n)
      load(ra, k + 1, 0);
    if (whole) {
      four(rb, 1);
    } else {  // the ragged top tile
#pragma unroll 1
      for (int j = 0; j < (int)S - base; ++j) {
        const int o = kFwd ? j : (int)S - base - 1 - j;
        step(o, sm.e[slot][lane * kRowF4 + o], sm.t[slot][o], out[o]);
      }
    }
    __syncwarp();
    // the tile's vectors leave together
    if ((uint32_t)base + unit < S) {
#pragma unroll
      for (uint32_t i = 0; i < 8; ++i)
        if (r0 + 4 * i <= last)
          beta[(size_t)(r0 + 4 * i) * S + (uint32_t)base + unit] =
              sm.v[slot][(r0 + 4 * i) * kRowF4 + unit];
    }
  }
  cp_async_wait<0>();
  __syncwarp();
}

// The recursions of a block's 32 samples, warp 0 the backward and warp 1 the forward
// one.  True for every thread once a sum was outside the fast reciprocal's range
// (never with kSafe): one below it left NaN in seen, one above it zeros, and with
// them such a sum or no unit sum at a half's end.
template <bool kSafe>
__device__ __forceinline__ bool chains_run(const GenParams &p, uint32_t s0, uint4 q) {
  extern __shared__ __align__(16) unsigned char glp_chain_smem[];
  ChainTiles *const tiles = reinterpret_cast<ChainTiles *>(glp_chain_smem);  // 0 backward
  const uint32_t lane = threadIdx.x & 31u;
  const bool fwd = threadIdx.x >= 32;
  const int n = ((int)p.S + kChainTile - 1) / kChainTile, n_lo = n / 2, n_hi = n - n_lo;
  float seen = 0.f;
  States v = fwd ? States{dup2(0.25f), dup2(0.25f)} : States{dup2(1.f), dup2(1.f)};
  auto special = [&]() {
    return !kSafe && !(seen == 0.f && v.P.x + v.P.y + v.Q.x + v.Q.y > 0.5f);
  };
  if (fwd)
    chain_run<true, false, kSafe>(p, tiles[1], lane, s0, q, v, seen, 0, n_lo);
  else
    chain_run<false, false, kSafe>(p, tiles[0], lane, s0, q, v, seen, kChainTile * (n - 1), n_hi);
  if (__syncthreads_or(special()))  // both halves' vectors are stored
    return true;
  if (fwd)
    chain_run<true, true, kSafe>(p, tiles[1], lane, s0, q, v, seen, kChainTile * n_lo, n_hi);
  else
    chain_run<false, true, kSafe>(p, tiles[0], lane, s0, q, v, seen, kChainTile * (n_lo - 1),
                                  n_lo);
  return __syncthreads_or(special()) != 0;
}

// A block's samples s0 .. s0 + 31 of one chunk.  A block with a sum outside the fast
// reciprocal's range starts over; the first halves cover every site, so it mostly
// shows at the middle.  With such a site in every block hmm_work takes 0.187 ms for
// 0.117 at 40 x 1,024, 0.207 for 0.129 at 2,000 x 1,024 and 0.73 for 0.53 at 10,000 x
// 2,048 (by one warp, its rows not staged, it took 1.16, 1.79 and 5.2).  Both forms
// are inlined: as a function of its own the second took a third longer.
__device__ __forceinline__ void work_chains(const GenParams &p, uint32_t s0) {
  const uint32_t s = min(s0 + (threadIdx.x & 31u), p.N - 1);
  const uint4 q = make_uint4(p.quad_out[s], p.quad_out[p.N + s], p.quad_out[2 * (size_t)p.N + s],
                             p.quad_out[3 * (size_t)p.N + s]);
  if (chains_run<false>(p, s0, q))
    chains_run<true>(p, s0, q);
}

inline __device__ __noinline__ float4 pow4(const float4 c, float pen) {
  return make_float4(powf(c.x, pen), powf(c.y, pen), powf(c.z, pen), powf(c.w, pen));
}

// Pass 2 of hmm_work: the sampling of impute.cpp:453-484 for site m of
// sample s, from p_m (pass 1), the genotype probabilities, the
// mutation-matrix rows pcr (pc[i][0..3] as float4) and the site's uniform
// u_bits (the draw's 32 bits; the trace's value when one is given).  Returns
// the two haplotype bits of the site as bits 0 and 1 (0 for sites past S).
__device__ __forceinline__ uint32_t work_sample_site(const GenParams &p, const float4 *pcr,
                                                     uint32_t s, uint32_t m, uint64_t A0,
                                                     uint64_t A1, uint64_t C0, uint64_t C1,
                                                     uint32_t u_bits) {
  const uint32_t S = p.S;
  if (m >= S)
    return 0;
  const uint32_t sh = m & 63u;
  const uint32_t a0 = (uint32_t)(A0 >> sh) & 1u, a1 = (uint32_t)(A1 >> sh) & 1u,
                 c0b = (uint32_t)(C0 >> sh) & 1u, c1b = (uint32_t)(C1 >> sh) & 1u;
  const States pp = states_of(__ldg(p.beta + (size_t)s * S + m));
  const float *pr = p.prob + ((size_t)s * S + m) * 3;
  const float g0 = __ldg(pr), g1 = __ldg(pr + 1), g2 = __ldg(pr + 2);
  const float4 r00 = pcr[(a0 << 1) | c0b], r01 = pcr[(a0 << 1) | c1b],
               r10 = pcr[(a1 << 1) | c0b], r11 = pcr[(a1 << 1) | c1b];
  const float2 p00 = dup2(pp.P.x), p01 = dup2(pp.P.y), p10 = dup2(pp.Q.y), p11 = dup2(pp.Q.x);
  // ((p00 r00 + p01 r01) + p10 r10) + p11 r11, two columns at a time
  auto inner = [&](float2 a, float2 b, float2 c, float2 d) {
    return add_pair(add_pair(add_pair(__fmul2_rn(p00, a), __fmul2_rn(p01, b)),
                                 __fmul2_rn(p10, c)),
                      __fmul2_rn(p11, d));
  };
  const float2 i01 = inner(make_float2(r00.x, r00.y), make_float2(r01.x, r01.y),
                           make_float2(r10.x, r10.y), make_float2(r11.x, r11.y));
  const float2 i23 = inner(make_float2(r00.z, r00.w), make_float2(r01.z, r01.w),
                           make_float2(r10.z, r10.w), make_float2(r11.z, r11.w));
  const float2 c01 = __fmul2_rn(make_float2(g0, g1), i01),
               c23 = __fmul2_rn(make_float2(g1, g2), i23);
  float4 c = make_float4(c01.x, c01.y, c23.x, c23.y);
  if (p.pen != 1.0f)
    c = pow4(c, p.pen);
  const float u = p.tr_work ? __ldg(p.tr_work + (size_t)s * S + m) : glp_u24(u_bits);
  const float s01 = __fadd_rn(c.x, c.y);
  const float s012 = __fadd_rn(s01, c.z);
  const float r = __fmul_rn(u, __fadd_rn(s012, c.w));
  // (0, 0), (0, 1), (1, 0), (1, 1)
  return r < c.x ? 0u : r < s01 ? 2u : r < s012 ? 1u : 3u;
}

// Pass 2 for words [w_lo, w_hi) of sample s (called by a whole warp; w_lo
// even), two words at a time: lane l draws the four uniforms of the l-th
// 4-site group of the
// 128-site span (one draw per group, as the reference draws them) into
// u[4 l .. 4 l + 3], so u[o] is the uniform of span site o; then the bits
// of sites w*64 + lane and w*64 + 32 + lane of each word are gathered into
// the two new haplotype words with ballots.
__device__ __forceinline__ void work_sample(const GenParams &p, const float4 *pcr, uint32_t s,
                                            uint4 q, uint32_t lane, uint32_t *u, uint32_t w_lo,
                                            uint32_t w_hi) {
  const uint32_t wn = p.wn;
  const uint64_t *f0 = p.haps + (size_t)q.x * wn, *f1 = p.haps + (size_t)q.y * wn,
                 *m0 = p.haps + (size_t)q.z * wn, *m1 = p.haps + (size_t)q.w * wn;
  uint64_t *ha = p.hnew + (size_t)2 * s * wn, *hb = ha + wn;
  for (uint32_t w2 = w_lo; w2 < w_hi; w2 += 2) {
    if (!p.tr_work) {
      const glp_u32x4 ux = glp_draw(p.seed, p.generation, s, 16 * w2 + lane, GLP_TAG_WORK);
      reinterpret_cast<uint4 *>(u)[lane] = make_uint4(ux.v[0], ux.v[1], ux.v[2], ux.v[3]);
    }
    __syncwarp();
#pragma unroll
    for (uint32_t t = 0; t < 2; ++t) {
      const uint32_t w = w2 + t;
      if (w >= w_hi)
        break;
      const uint64_t A0 = __ldg(f0 + w), A1 = __ldg(f1 + w), C0 = __ldg(m0 + w),
                     C1 = __ldg(m1 + w);
      const uint32_t lo = work_sample_site(p, pcr, s, w * 64 + lane, A0, A1, C0, C1,
                                           u[64 * t + lane]);
      const uint32_t hi = work_sample_site(p, pcr, s, w * 64 + 32 + lane, A0, A1, C0, C1,
                                           u[64 * t + 32 + lane]);
      const uint32_t alo = __ballot_sync(0xffffffffu, lo & 1u),
                     ahi = __ballot_sync(0xffffffffu, hi & 1u);
      const uint32_t blo = __ballot_sync(0xffffffffu, lo & 2u),
                     bhi = __ballot_sync(0xffffffffu, hi & 2u);
      if (lane == 0) {
        ha[w] = ((uint64_t)ahi << 32) | alo;
        hb[w] = ((uint64_t)bhi << 32) | blo;
      }
    }
    __syncwarp();  // u is redrawn next span
  }
}

// ---------------------------------------------------------------------------
// The generation kernels.

__device__ __forceinline__ void set_slot(uint4 &q, uint32_t r, uint32_t v) {
  if (r == 0)
    q.x = v;
  else if (r == 1)
    q.y = v;
  else if (r == 2)
    q.z = v;
  else
    q.w = v;
}

// Speculation trees.  A round of n evaluations scores n nodes of the tree of a
// chain's possible decisions: the root is the chain's next position, a node's two
// children the position after it with the node's proposal refused or accepted.  At
// an acceptance rate a the n nodes most likely to be reached -- a node's chance is
// the product of a or 1 - a along its path -- are a line of refusals for a small
// a, a line of acceptances for a near 1, and branched between: with 16 nodes the
// chain goes on 7.3 positions a round at a = 0.12, 4.3 at 0.35 (2.9 on a line of
// refusals), 12 at 0.96 (1.0).  The nodes are numbered in the order in which a
// greedy search takes them, so that a tree's first n nodes are the tree for n.
// Which nodes are scored changes no result: each is the evaluation that the chain
// would make there, and the chain takes those on its way.  A generation of few
// chains lasts as long as the chain that accepts most often: 3 x 3 0.183 and 0.108
// ms, 256 x 1,024 0.559 and 0.532, 30 generations of 60 x 1,000 17.6 and 16.7.
struct SpecNode {
  uint32_t path;    // its ancestors: bit 2 i for node i
  uint32_t accept;  // those of them whose proposal it has accepted
  uint32_t desc;    // [0, 4) depth, [4, 8) the last of those, [8, 24) their depths
};
struct SpecTrees {
  SpecNode node[kSpecRates][kSpecNodes];
};
constexpr SpecTrees make_spec_trees() {
  SpecTrees t{};
  for (int i = 0; i < kSpecRates; ++i) {
    const SpecShape sh = make_spec_shape(i);
    for (int n = 1; n < kSpecNodes; ++n) {
      const int from = sh.parent[n];
      const bool dec = sh.accept[n];
      const SpecNode &pa = t.node[i][from];
      const uint32_t depth = pa.desc & 15u;
      SpecNode &nd = t.node[i][n];
      nd.path = pa.path | (1u << (2 * from));
      nd.accept = pa.accept | (dec ? 1u << (2 * from) : 0u);
      nd.desc = (depth + 1) | (dec ? (uint32_t)from << 4 : pa.desc & 0xf0u) |
                (pa.desc & 0xffff00u) | (dec ? 0x100u << depth : 0u);
    }
  }
  return t;
}
static __device__ const SpecTrees kSpecTrees = make_spec_trees();
// The same for the nodes of a team: node 16 w + i is bit 2 i of word w.
struct __align__(16) TeamNode {
  uint32_t path[4], accept[4];
  uint32_t taken[2];  // the accepted ancestors' depths
  uint32_t desc;      // [0, 8) depth, [8, 16) the last of those
  uint32_t unused;
};
struct TeamTrees {
  TeamNode node[kSpecRates][kTeamNodes];
};
constexpr TeamTrees make_team_trees() {
  TeamTrees t{};
  for (int i = 0; i < kSpecRates; ++i) {
    const SpecShape sh = make_spec_shape(i);
    for (int n = 1; n < kTeamNodes; ++n) {
      const int from = sh.parent[n];
      const bool dec = sh.accept[n];
      TeamNode &nd = t.node[i][n];
      nd = t.node[i][from];
      const uint32_t depth = nd.desc & 255u, bit = 1u << (2 * (from % kSpecNodes));
      nd.path[from / kSpecNodes] |= bit;
      if (dec) {
        nd.accept[from / kSpecNodes] |= bit;
        nd.taken[depth / 32] |= 1u << (depth % 32);
        nd.desc = (uint32_t)from << 8;
      }
      nd.desc = (nd.desc & 0xff00u) | (depth + 1);
    }
  }
  return t;
}
static __device__ const TeamTrees kTeamTrees = make_team_trees();
// A chain's rate moves with weight 1 / 24 a cycle from the generation's (with 1 / 6,
// chains of 10,000 samples took 0.8 % more rounds, 3 x 3 sites 1 % fewer).
constexpr float kRateWeight = 24.0f;
// The accept rule compares a uniform u with a float f: f > u for a float f exactly
// when f > bound, and u = 0 has the bound -0.
__device__ __forceinline__ float accept_bound(double u) {
  return u == 0.0 ? -0.0f : __double2float_rd(u);
}

// One cycle's draws: the accept uniform, the proposed haplotype and the slot that
// it replaces.
struct __align__(16) Draw {
  float u;  // accept_bound
  uint32_t hap, slot, unused;
};
constexpr uint32_t kDraws = 64;  // a warp's windows: two per lane of each group

__device__ __forceinline__ Draw make_draw(const GenParams &p, uint32_t s, uint32_t cyc,
                                          int *error) {
  Draw d;
  double u;
  if (p.tr_slot) {
    d.slot = p.tr_slot[(size_t)s * p.C + cyc] & 3u;
    u = p.tr_u[(size_t)s * p.C + cyc];
  } else {
    glp_mh_draw(p.seed, p.generation, s, cyc, &d.slot, &u);
  }
  d.u = accept_bound(u);
  d.hap = p.props ? __ldg(p.props + (size_t)cyc * p.N + s)
          : (p.kick_first && cyc == 0)
              ? glp_surrogate_ref(p.seed, p.generation, s, cyc, GLP_TAG_PROP, 2u * p.N, p.H,
                                  p.nbr, p.klen)
              : glp_surrogate(p.seed, p.generation, s, cyc, GLP_TAG_PROP, p.samp_lo, p.samp_hi,
                              p.nbr, p.klen);
  if (d.hap >= p.H) {
    atomicOr(error, 1);
    d.hap = 0;
  }
  return d;
}

// The accepted ancestors' haplotypes into q, whose slots in `have` are set: from
// the last, at the highest of the bits of m (the draws of the cycles from `first`
// on), to the first that still finds its slot open.
__device__ __forceinline__ void place_path(uint4 &q, const Draw *window, uint32_t wmask,
                                           uint32_t first, uint32_t m, uint32_t &have) {
  while (m != 0u && have != 15u) {
    const uint32_t top = 31u - __clz(m);
    const Draw d = window[(first + top) & wmask];
    if (!((have >> d.slot) & 1u)) {
      set_slot(q, d.slot, d.hap);
      have |= 1u << d.slot;
    }
    m ^= 1u << top;
  }
}

// Work sources.  One chunk: the kernel parameter.  Many chunks: a descriptor
// table in global memory; the samples of all chunks form one queue, chunk by
// chunk, so a group's neighbours in the queue usually share its chunk.
// Pass 2 splits each sample's words into parts of kSampleWords, one warp a
// part, so that its warps are many and short and the last of them leave little
// of the GPU idle.
#ifndef GLP_SAMPLE_WORDS
#define GLP_SAMPLE_WORDS 16
#endif
constexpr uint32_t kSampleWords = GLP_SAMPLE_WORDS;
static_assert(kSampleWords % 2 == 0, "a part starts a two-word span");
__host__ __device__ inline uint32_t sample_parts(uint32_t wn) {
  return (wn + kSampleWords - 1) / kSampleWords;
}

struct OneChunk {
  static constexpr bool kMulti = false;
  const GenParams &p;
  __device__ __forceinline__ uint32_t total() const { return p.N; }
  __device__ __forceinline__ const GenParams &chunk(uint32_t) const { return p; }
  __device__ __forceinline__ void locate(uint32_t g, uint32_t &c, uint32_t &s) const {
    c = 0;
    s = g;
  }
  __device__ __forceinline__ void locate_block(uint32_t b, uint32_t &c, uint32_t &s0) const {
    c = 0;
    s0 = b * kChainSamples;
  }
  __device__ __forceinline__ void locate_part(uint32_t g, uint32_t &c, uint32_t &s,
                                              uint32_t &part) const {
    const uint32_t parts = sample_parts(p.wn);
    c = 0;
    s = g / parts;
    part = g % parts;
  }
};

// Device tables of a batch of n chunks, one array of batch_words(n) words:
//   [0, n]            prefix sums of the chunks' N in the order that follows (the
//                     generation kernel's queue)
//   [n + 1, 2n]       the chunks in order of falling S (the longest chains and
//                     recursions start first: a generation of the eight chunks 14.05
//                     ms in the caller's order, 13.3 in this)
//   [2n + 1, 3n + 1]  in that order, prefix sums of the blocks of hmm_work's
//                     pass 1 (ceil(N / kChainSamples) each)
//   [3n + 2, 4n + 2]  in that order, prefix sums of the warps of its pass 2
//                     (N sample_parts(wn) each)
// Chunks without hmm_work have no blocks and no warps.
__host__ __device__ inline size_t batch_words(uint32_t n) { return 4 * (size_t)n + 3; }

struct MultiParams {
  const GenParams *chunks;   // [nchunks]
  const uint32_t *offsets;   // the tables above
  uint32_t nchunks;
  uint32_t *counter;
  unsigned long long *stats;
  int *error;
};

struct ManyChunks {
  static constexpr bool kMulti = true;
  const MultiParams &mp;
  __device__ __forceinline__ uint32_t total() const { return __ldg(mp.offsets + mp.nchunks); }
  __device__ __forceinline__ const GenParams &chunk(uint32_t c) const { return mp.chunks[c]; }
  // largest i < nchunks with prefix[i] <= g
  __device__ __forceinline__ uint32_t find(const uint32_t *prefix, uint32_t g) const {
    uint32_t lo = 0, hi = mp.nchunks;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(prefix + mid) <= g)
        lo = mid;
      else
        hi = mid;
    }
    return lo;
  }
  __device__ __forceinline__ void locate(uint32_t g, uint32_t &c, uint32_t &s) const {
    const uint32_t i = find(mp.offsets, g);
    c = __ldg(mp.offsets + mp.nchunks + 1 + i);
    s = g - __ldg(mp.offsets + i);
  }
  __device__ __forceinline__ void locate_block(uint32_t b, uint32_t &c, uint32_t &s0) const {
    const uint32_t *order = mp.offsets + mp.nchunks + 1, *blocks = order + mp.nchunks;
    const uint32_t i = find(blocks, b);
    c = __ldg(order + i);
    s0 = (b - __ldg(blocks + i)) * kChainSamples;
  }
  __device__ __forceinline__ void locate_part(uint32_t g, uint32_t &c, uint32_t &s,
                                              uint32_t &part) const {
    const uint32_t *order = mp.offsets + mp.nchunks + 1,
                   *warps = order + 2 * mp.nchunks + 1;
    const uint32_t i = find(warps, g);
    c = __ldg(order + i);
    const uint32_t parts = sample_parts(mp.chunks[c].wn);
    s = (g - __ldg(warps + i)) / parts;
    part = (g - __ldg(warps + i)) % parts;
  }
};

// Lane groups of a warp.  A warp starts as 32/P groups of P lanes (P is the
// smallest group size the kernel is instantiated for).  Once the sample queue
// is exhausted and some of the warp's groups have no sample left, the warp's
// 32 lanes are re-partitioned among its remaining samples: na samples get
// groups of p = 32 / nextpow2(na) or 2p lanes (the 2p-groups first, every
// group aligned to its size), so the longest chains of a generation finish
// with wider speculation instead of leaving lanes idle.
struct LaneGroups {
  uint32_t size, base, index, count;
};

__device__ __forceinline__ LaneGroups regroup(uint32_t lane, uint32_t na) {
  const uint32_t np2 = 1u << (32 - __clz(na - 1u));  // nextpow2(na), na >= 1
  const uint32_t p = 32u / (na > 1 ? np2 : 1u);
  const uint32_t nbig = 32u / p - na;  // groups of 2p lanes
  LaneGroups g;
  g.count = na;
  if (lane < nbig * 2 * p) {
    g.size = 2 * p;
    g.index = lane / (2 * p);
    g.base = g.index * 2 * p;
  } else {
    g.size = p;
    g.index = nbig + (lane - nbig * 2 * p) / p;
    g.base = nbig * 2 * p + (g.index - nbig) * p;
  }
  return g;
}

// The accept rule of MHSampler<T>::SampleHap (MHSampler.hpp:86-93) for a
// uniform u in [0, 1) with 53-bit resolution: accept when prop >= curr or
// u < exp((prop - curr) pen).  For d = (prop - curr) pen in (-37, 0) the
// exponential is taken in binary32 (relative error below 3e-6: a decision can
// differ from the binary64 one only where |d - ln u| < 3e-6); below -37 it
// is under 2^-53, so only u = 0 accepts, as in binary64.
// u comes as accept_bound(u).
__device__ __forceinline__ bool mh_accept(double prop, double curr, double pen, float bound) {
  if (prop >= curr)
    return true;
  const double d = (prop - curr) * pen;
  if (d > -37.0)
    return expf((float)d) > bound;
  return __float_as_uint(bound) == 0x80000000u && exp(d) > 0.0;
}

// The quadruple that sample s starts a generation with.
__device__ __forceinline__ uint4 first_quad(const GenParams &p, uint32_t s, int *error) {
  const uint32_t N = p.N, H = p.H;
  uint4 q;
  if (p.quad_in) {
    q = make_uint4(__ldg(p.quad_in + s), __ldg(p.quad_in + N + s),
                   __ldg(p.quad_in + 2 * (size_t)N + s), __ldg(p.quad_in + 3 * (size_t)N + s));
  } else {
    // fresh quadruple from the sampler, as RunHMMOnSamples draws one
    // every generation (hmmLike.cpp:90-95)
    q.x = glp_surrogate(p.seed, p.generation, s, 0, GLP_TAG_INIT, p.samp_lo, p.samp_hi, p.nbr,
                        p.klen);
    q.y = glp_surrogate(p.seed, p.generation, s, 1, GLP_TAG_INIT, p.samp_lo, p.samp_hi, p.nbr,
                        p.klen);
    q.z = glp_surrogate(p.seed, p.generation, s, 2, GLP_TAG_INIT, p.samp_lo, p.samp_hi, p.nbr,
                        p.klen);
    q.w = glp_surrogate(p.seed, p.generation, s, 3, GLP_TAG_INIT, p.samp_lo, p.samp_hi, p.nbr,
                        p.klen);
  }
  if (q.x >= H || q.y >= H || q.z >= H || q.w >= H) {
    atomicOr(error, 1);
    q = make_uint4(0, 0, 0, 0);
  }
  return q;
}

template <int P, class E, class Src, int kSub = 1>
__device__ __forceinline__ void generation_body(const Src &src, uint32_t *counter,
                                                unsigned long long *stats, int *error,
                                                const float4 *vq_smem) {
  static_assert(P == 2 || P == 4 || P == 8 || P == 16 || P == 32, "P");
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t G0 = 32u / P;  // group slots (staging rings) per warp
  constexpr bool kTree = kSpecTree(P);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  // current partition of the warp's lanes
  uint32_t Pc = P, gbase = lane - lane % P, gidx = lane / P, ngroups = G0;
  uint32_t li = lane - gbase;
  // kWarps * (32/P) * kGroupStrideF4 float4 of rings, then the warps' draws
  extern __shared__ float4 glp_stage[];
  Draw *const draws = reinterpret_cast<Draw *>(glp_stage + (size_t)kWarps * G0 * kGroupStrideF4) +
                      warp * kDraws;
  uint32_t drawn = 0;  // cycles of the sample whose draws the window has reached

  const uint32_t total = src.total();
  // The first samples are dealt out evenly over the warps: sample g * W + w of the
  // queue to group slot g of global warp w, or in a batch neighbours in the queue
  // to a warp, which are of one chunk mostly, so that the warp's groups run in step
  // (eight chunks of 4,416 to 8,192 sites 13.3 and 13.1 ms; 2,000 x 8,192 is 5 %
  // slower so).  Later samples come from the queue counter, offset past those.
  const uint32_t nwarps = gridDim.x * (uint32_t)kWarps;
  const uint32_t gwarp = blockIdx.x * (uint32_t)kWarps + warp;
  const uint32_t spread = (uint32_t)min((unsigned long long)total,
                                        (unsigned long long)G0 * nwarps);
  const uint32_t share = spread / nwarps, extra = spread % nwarps;
  const uint32_t dealt = share + (gwarp < extra ? 1u : 0u);
  const uint32_t from0 = Src::kMulti ? gwarp * share + min(gwarp, extra) : gwarp,
                 step = Src::kMulti ? 1u : nwarps;
  bool first = true;
  uint32_t c = 0, s = kNone, e = 0;
  uint4 q = make_uint4(0, 0, 0, 0);
  double curr = 0.0;
  float rate = 0.0f;  // the chain's acceptance rate so far
  bool exhausted = false;
  unsigned long long n_evals = 0, n_rounds = 0, n_acc = 0;
  unsigned long long n_warp_rounds = 0, n_active_lanes = 0;

  while (true) {
    // idle groups take the next sample from the generation's queue
    const bool need = (s == kNone) && !exhausted;
    uint32_t ns = 0;
    if (need && li == 0) {
      if (first) {
        ns = gidx < dealt ? from0 + gidx * step : total;
      } else {
        ns = spread + atomicAdd(counter, 1u);
      }
    }
    first = false;
    ns = __shfl_sync(FULL, ns, gbase);
    if (need) {
      if (ns < total) {
        src.locate(ns, c, s);
        e = 0;
        drawn = 0;
        const GenParams &p = src.chunk(c);
        if (kTree)
          rate = p.rate;
        q = first_quad(p, s, error);
      } else {
        exhausted = true;
      }
    }
    // groups still without a sample cannot get one any more: hand their
    // lanes to the warp's remaining samples
    const unsigned lead = __ballot_sync(FULL, li == 0 && s != kNone);
    if (lead == 0)
      break;
    const uint32_t na = __popc(lead);
    if (na < ngroups) {
      const LaneGroups ng = regroup(lane, na);
      const uint32_t from = __fns(lead, 0, (int)ng.index + 1);
      c = __shfl_sync(FULL, c, from);
      s = __shfl_sync(FULL, s, from);
      e = __shfl_sync(FULL, e, from);
      q.x = __shfl_sync(FULL, q.x, from);
      q.y = __shfl_sync(FULL, q.y, from);
      q.z = __shfl_sync(FULL, q.z, from);
      q.w = __shfl_sync(FULL, q.w, from);
      curr = __shfl_sync(FULL, curr, from);
      if (kTree)
        rate = __shfl_sync(FULL, rate, from);
      Pc = ng.size;
      gbase = ng.base;
      gidx = ng.index;
      ngroups = ng.count;
      li = lane - gbase;
      exhausted = true;
      drawn = max(e, 1u) - 1;  // the window lies elsewhere now
    }
    const bool active = s != kNone;
    const unsigned amask = __ballot_sync(FULL, active);
    if (lane == 0) {
      ++n_warp_rounds;
      n_active_lanes += __popc(amask);
    }

    const GenParams &p = src.chunk(c);
    const uint32_t N = p.N, C = p.C, H = p.H;
    // One speculative round: the group's Pc/2 lane pairs score the first Pc/2
    // nodes of the speculation tree for the chain's rate, pair r = li/2 node r, at
    // position e + depth (its even lane the forward half, its odd lane the
    // backward half of the evaluation).  Position 0 is the quadruple that the
    // chain starts with, neither accepted nor refused: the round that begins there
    // takes the line of refusals, as every round of a narrow kernel does.
    const uint32_t npos = Pc >> 1, r = li >> 1;
    uint32_t path = 0, wants = 0, desc = r;
    if (kTree) {
      const uint32_t tree = e == 0 ? 0u : (uint32_t)(rate * 16.0f + 0.5f);
      const SpecNode *const node = &kSpecTrees.node[min(tree, kSpecRates - 1u)][r];
      path = __ldg(&node->path);
      wants = __ldg(&node->accept);
      desc = __ldg(&node->desc);
    }
    const uint32_t depth = desc & 15u, taken = desc >> 8, ev = e + depth;
    const bool lead_lane = (li & 1u) == 0;
    const uint32_t k = active ? min(npos, C + 1 - e) : 0u;  // positions, at most
    const bool valid = depth < k, scores = valid && ev > 0;
    // Draws of cycle i at entry i mod 2 Pc of the group's window, made Pc cycles
    // at a time, one a lane, when the window does not reach this round's last one
    // (or another group of the warp draws and there is room): a chain makes each
    // draw once, and the other rounds only read them.  The generators' chain of
    // integer products stood in front of every round (3 x 3 0.241 and 0.214 ms, 3,001
    // x 4,000 from codes 4.52 and 4.45, 2,000 x 8,192 5.72 and 5.58).  The first words
    // of the proposals' rows are not asked for ahead: that was never faster (256 x
    // 1,024 at 64 lanes 0.296 and without it 0.292, 2,000 x 2,048 1.076 and 1.072), and
    // where all warps ask for the same few lines, as neighbour lists over few sites
    // make them, slow (584 x 9 at 64 lanes 0.123 and 0.075).
    Draw *const window = draws + 2 * gbase;
    const uint32_t wmask = 2 * Pc - 1, next = max(e, 1u) - 1;  // the round's first cycle
    if (__any_sync(FULL, active && drawn < min(C, e + k - 1))) {
      if (active && drawn < C && drawn + Pc - next <= 2 * Pc) {
        const uint32_t cyc = drawn + li;
        if (cyc < C) {
          const Draw d = make_draw(p, s, cyc, error);
          window[cyc & wmask] = d;
        }
        drawn += Pc;
      }
      __syncwarp();
    }
    uint32_t slot = 0, phap = 0;
    float u = 0.0f;
    uint4 myq = q;
    if (scores) {
      const Draw d = window[(ev - 1) & wmask];
      slot = d.slot;
      phap = d.hap;
      u = d.u;
      set_slot(myq, slot, phap);
      if (kTree && taken) {
        uint32_t have = 1u << slot;
        place_path(myq, window, wmask, e - 1, taken, have);
      }
    }
    double L = 0.0;
    // When every lane of the warp scores a chunk of the same length, all
    // groups run the same block loop and synchronise as one warp: a
    // group-masked __syncwarp would let the groups drift apart and issue the
    // loop body once per group.
    unsigned same = 0;
    __match_all_sync(FULL, active ? p.S : 0u, (int *)&same);
    const bool warp_lockstep = same && amask == FULL;
    if (active) {
      // every pair of an active group evaluates (positions past k score the
      // base quadruple and drop the result) so the group shares its ring
      E em;
      em.init(p, s, Src::kMulti ? p.vq_table : vq_smem);
      const unsigned gm = (Pc == 32 || warp_lockstep) ? FULL : (((1u << Pc) - 1u) << gbase);
      float4 *ring = glp_stage + ((size_t)warp * G0 + gidx) * kGroupStrideF4;
      L = (gm == FULL)
              ? eval_pair<(P >= 8 ? 1 : 8 / P), E, kSub, true, P == 8>(p, em, myq, ring, li, Pc,
                                                                       gm)
              : eval_pair<(P >= 8 ? 1 : 8 / P), E, kSub, false, P == 8>(p, em, myq, ring, li,
                                                                        Pc, gm);
      if (!valid)
        L = 0.0;
    }
    const double pen = (double)p.pen;
    const double L0 = __shfl_sync(FULL, L, gbase);
    const double curr0 = (e == 0) ? L0 : curr;
    if constexpr (kTree) {
      // The accept rule of MHSampler.hpp:86-93.  Every node's test is made at once,
      // against the likelihood that is current on its path: that of the last node
      // accepted there, or the round's first.  The chain reaches the nodes whose
      // ancestors decided as their paths say, the deepest of them the last in number:
      // the same decisions as the sequential loop.  The even lanes vote.
      const double Lup = __shfl_sync(FULL, L, gbase + 2u * ((desc >> 4) & 15u));
      const bool acc = lead_lane && scores && mh_accept(L, taken ? Lup : curr0, pen, u);
      const uint32_t gones = Pc == 32 ? FULL : (1u << Pc) - 1u;
      const unsigned abal = (__ballot_sync(FULL, acc) >> gbase) & gones;
      const bool hit = lead_lane && valid && ((abal ^ wants) & path) == 0u;
      unsigned reached = (__ballot_sync(FULL, hit) >> gbase) & gones;
      const unsigned accepted = abal & reached;
      const uint32_t end = active ? 31u - __clz(reached) : 0u;  // twice the last node
      const uint32_t la = accepted ? 31u - __clz(accepted) : 0u;
      double cur = __shfl_sync(FULL, L, gbase + la);
      const uint4 qa = make_uint4(
          __shfl_sync(FULL, myq.x, gbase + la), __shfl_sync(FULL, myq.y, gbase + la),
          __shfl_sync(FULL, myq.z, gbase + la), __shfl_sync(FULL, myq.w, gbase + la));
      // Where the chain accepts at its last node, the nodes on that one's line of
      // refusals that replace the same slot scored exactly the quadruple that the
      // chain builds there, so the chain goes on through them -- each tested against
      // the likelihood accepted last -- up to the first that replaces another slot.
      const uint32_t desc_e = __shfl_sync(FULL, desc, gbase + end);
      const uint32_t slot_e = __shfl_sync(FULL, slot, gbase + end);
      const bool line = lead_lane && valid && taken == desc_e >> 8 && depth > (desc_e & 15u);
      unsigned run = (__ballot_sync(FULL, line) >> gbase) & gones;
      const unsigned other = (__ballot_sync(FULL, line && slot != slot_e) >> gbase) & gones;
      if (!accepted || la != end)
        run = 0;
      else if (other)
        run &= (other & (0u - other)) - 1u;
      uint32_t hap = 0;
      unsigned more = 0;  // accepted nodes of the run
      reached |= run;
      while (__any_sync(FULL, run != 0u)) {
        const uint32_t from = gbase + (run ? (uint32_t)__ffs(run) - 1u : 0u);
        const double L_r = __shfl_sync(FULL, L, from);
        const float u_r = __shfl_sync(FULL, u, from);
        const uint32_t ph_r = __shfl_sync(FULL, phap, from);
        if (run) {
          if (mh_accept(L_r, cur, pen, u_r)) {
            cur = L_r;
            hap = ph_r;
            more |= run & (0u - run);
          }
          run &= run - 1u;
        }
      }
      if (active) {
        curr = curr0;
        if (accepted) {
          curr = cur;
          q = qa;
          if (more)
            set_slot(q, slot_e, hap);
        }
      }
      const unsigned mine = 1u << (lane - gbase);
      if (lead_lane && (reached & mine)) {
        if (p.eval_trace)
          p.eval_trace[(size_t)s * (C + 1) + ev] = L;
        if (ev > 0 && p.accept_trace)
          p.accept_trace[(size_t)s * C + ev - 1] = (uint8_t)(((accepted | more) & mine) != 0u);
      }
      const uint32_t scored =
          (uint32_t)__popc((__ballot_sync(FULL, lead_lane && valid) >> gbase) & gones);
      if (active) {
        const uint32_t steps = (uint32_t)__popc(reached),
                       na = (uint32_t)(__popc(accepted) + __popc(more));
        rate = __fdividef(kRateWeight * rate + (float)na,
                          kRateWeight + (float)(steps - (e == 0 ? 1u : 0u)));
        e += steps;
        if (li == 0) {
          n_evals += scored;
          ++n_rounds;
          n_acc += na;
        }
      }
    } else {
      // The accept rule of MHSampler.hpp:86-93 in chain order.  Every
      // evaluation of the round was built on the round's starting state, and
      // until the first acceptance the chain's current likelihood is the
      // starting one, so each position tests its own proposal against it in
      // parallel and the first accepting position (in chain order) wins: the
      // same decisions as the sequential loop.  The even lanes vote.
      const bool acc = lead_lane && r < k && ev > 0 && mh_accept(L, curr0, pen, u);
      const unsigned gmask = (Pc == 32) ? FULL : (((1u << Pc) - 1u) << gbase);
      const unsigned abal = __ballot_sync(FULL, acc) & gmask;
      const uint32_t srcl = abal ? (uint32_t)(__ffs(abal) - 1) : gbase;
      const uint32_t first_acc = abal ? (srcl - gbase) >> 1 : npos;
      const double La = __shfl_sync(FULL, L, srcl);
      const uint32_t sla = __shfl_sync(FULL, slot, srcl);
      const uint32_t pha = __shfl_sync(FULL, phap, srcl);
      // The positions after the first acceptance that replace the same slot
      // scored exactly the quadruple the sequential chain builds there (it
      // differs from the round's start only in that slot), so the chain goes on
      // through them -- each tested against the likelihood accepted last --
      // up to the first position that replaces another slot.
      uint32_t last = first_acc, hap = pha;
      uint32_t more = 0;  // accepted positions after first_acc
      double cur = La;
      const unsigned others = __ballot_sync(FULL, !(scores && lead_lane && slot == sla)) &
                              0x55555555u & gmask;
      // pairs after the first accepting one up to the next that replaces another slot
      const unsigned after = others & ~((2u << srcl) - 1u);
      const uint32_t stop =
          !abal ? 0u : after ? ((uint32_t)__ffs(after) - 1 - gbase) >> 1 : npos;
      for (uint32_t r2 = first_acc + 1; __any_sync(FULL, r2 < stop); ++r2) {
        const uint32_t from = gbase + 2u * (r2 < stop ? r2 : 0u);
        const double L_r = __shfl_sync(FULL, L, from);
        const float u_r = __shfl_sync(FULL, u, from);
        const uint32_t ph_r = __shfl_sync(FULL, phap, from);
        if (r2 < stop) {
          last = r2;
          if (mh_accept(L_r, cur, pen, u_r)) {
            cur = L_r;
            hap = ph_r;
            more |= 1u << r2;
          }
        }
      }
      if (active) {
        curr = curr0;
        if (abal) {
          set_slot(q, sla, hap);
          curr = cur;
        }
      }
      if (lead_lane && r < k && r <= last) {
        if (p.eval_trace)
          p.eval_trace[(size_t)s * (C + 1) + ev] = L;
        if (ev > 0 && p.accept_trace)
          p.accept_trace[(size_t)s * C + ev - 1] =
              (uint8_t)(r == first_acc || ((more >> r) & 1u));
      }
      if (active) {
        e = (first_acc < npos) ? e + last + 1 : e + k;
        if (li == 0) {
          n_evals += k;
          ++n_rounds;
          n_acc += first_acc < npos ? 1u + (uint32_t)__popc(more) : 0u;
        }
      }
    }

    // finished chains: publish (hmm_work samples their haplotypes)
    const bool done = active && e > C;
    if (done && li == 0) {
      p.quad_out[s] = q.x;
      p.quad_out[N + s] = q.y;
      p.quad_out[2 * (size_t)N + s] = q.z;
      p.quad_out[3 * (size_t)N + s] = q.w;
      if (p.like_out)
        p.like_out[s] = curr;
    }
    if (done)
      s = kNone;
  }
  if (stats && n_rounds) {  // per-lane counts of the rounds this lane led
    atomicAdd(stats, n_evals);
    atomicAdd(stats + 1, n_rounds);
    atomicAdd(stats + 2, n_acc);
  }
  if (stats && n_warp_rounds) {
    atomicAdd(stats + 4, n_warp_rounds);
    atomicAdd(stats + 5, n_active_lanes);
  }
}

// What the warps of a team show one another in a round, a warp's part.
struct __align__(16) TeamShare {
  uint4 q[kSpecNodes];
  double L[kSpecNodes];
  uint32_t accepts, reached, next, unused;
};

// Generations of few samples: W warps of a block score 16 W nodes of a chain's
// tree.  The chains are as long as before in evaluations and shorter in rounds (at
// a = 0.12 a round goes on 7.3, 8.8 and 10.6 positions with 16, 32 and 64 nodes), and
// the added warps run on schedulers that would stand idle.  Each warp stages the
// sample's rows for itself; the warps meet at four barriers a round: for the
// draws, the likelihoods, the votes and the nodes reached.  Where a round ends with an
// acceptance the chain starts its next one there: the tree has that child mostly.
// Measured, a team against one warp a chain: 60 x 1,024 0.351 and 0.234 ms (four
// warps), 256 x 1,024 0.356 and 0.265 (two), 100 x 8,192 2.55 and 1.47, 3 x 3 0.056
// and 0.041, 60 x 1,000 from codes 0.553 and 0.345.  Bound now: the chain of a site,
// by the rounds of the longest chain.
template <int W, class E, int kSub>
__device__ __forceinline__ void generation_team(const GenParams &p, const float4 *vq_smem) {
  static_assert(W == 2 || W == 4, "W");
  static_assert(kWarps % W == 0, "a block holds whole teams");
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t kNodes = (uint32_t)(kSpecNodes * W), kLanes = 32u * W;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, wt = warp % W,
                 team = warp / W;
  const uint32_t tl = 32 * wt + lane, r = tl >> 1;
  const bool lead_lane = (lane & 1u) == 0;
  extern __shared__ float4 glp_stage[];
  float4 *const ring = glp_stage + (size_t)warp * kGroupStrideF4;
  Draw *const window = reinterpret_cast<Draw *>(glp_stage + (size_t)kWarps * kGroupStrideF4) +
                       team * W * kDraws;
  TeamShare *const share =
      reinterpret_cast<TeamShare *>(glp_stage + (size_t)kWarps * (kGroupStrideF4 + kDraws)) +
      team * W;
  static_assert(kDraws * W == 2 * kLanes && sizeof(Draw) == sizeof(float4), "window");
  auto meet = [&]() {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kLanes) : "memory");
  };
  const uint32_t N = p.N, C = p.C, teams = gridDim.x * (uint32_t)(kWarps / W);
  const double pen = (double)p.pen;
  unsigned long long n_evals = 0, n_rounds = 0, n_acc = 0, n_warp_rounds = 0;

  for (uint32_t s = blockIdx.x * (uint32_t)(kWarps / W) + team; s < N;) {
    uint4 q = first_quad(p, s, p.error);
    double curr = 0.0;
    float rate = p.rate;
    uint32_t drawn = 0;
    E em;
    em.init(p, s, vq_smem);
    for (uint32_t e = 0; e <= C;) {
      const uint32_t tree = e == 0 ? 0u : (uint32_t)(rate * 16.0f + 0.5f);
      const TeamNode *const node = &kTeamTrees.node[min(tree, kSpecRates - 1u)][r];
      const uint32_t desc = __ldg(&node->desc), t0 = __ldg(&node->taken[0]),
                     t1 = __ldg(&node->taken[1]);
      const uint32_t depth = desc & 255u, ev = e + depth, k = min(kNodes, C + 1 - e);
      const bool valid = depth < k, scores = valid && ev > 0;
      // draws as in generation_body, for the team
      constexpr uint32_t wmask = 2 * kLanes - 1;
      if (drawn < min(C, e + k - 1)) {
        const uint32_t cyc = drawn + tl;
        if (cyc < C)
          window[cyc & wmask] = make_draw(p, s, cyc, p.error);
        drawn += kLanes;
      }
      // The draws are there.  And every warp has read what the last round shared: its
      // likelihoods, quadruples, votes and nodes reached are written over below, and
      // nothing but this barrier stands between.
      meet();
      uint4 myq = q;
      float u = 0.0f;
      if (scores) {
        const Draw d = window[(ev - 1) & wmask];
        u = d.u;
        set_slot(myq, d.slot, d.hap);
        if (t0 | t1) {
          uint32_t have = 1u << d.slot;
          place_path(myq, window, wmask, e + 31, t1, have);
          place_path(myq, window, wmask, e - 1, t0, have);
        }
      }
      const double L = eval_pair<1, E, kSub, true, false>(p, em, myq, ring, lane, 32, FULL);
      if (lead_lane) {
        share[wt].L[lane >> 1] = L;
        share[wt].q[lane >> 1] = myq;
      }
      meet();
      if (e == 0)
        curr = share[0].L[0];
      const uint32_t up = (desc >> 8) & 255u;
      const double at = (t0 | t1) ? share[up / kSpecNodes].L[up % kSpecNodes] : curr;
      const unsigned votes =
          __ballot_sync(FULL, lead_lane && scores && mh_accept(L, at, pen, u));
      if (lane == 0)
        share[wt].accepts = votes;
      meet();
      bool hit = lead_lane && valid;
#pragma unroll
      for (int w = 0; w < W; ++w)
        hit = hit && ((share[w].accepts ^ __ldg(&node->accept[w])) & __ldg(&node->path[w])) == 0u;
      const unsigned mine = __ballot_sync(FULL, hit);
      if (lane == 0)
        share[wt].reached = mine;
      meet();
      uint32_t steps = 0, na = 0, la = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const unsigned reached = share[w].reached, accepted = reached & share[w].accepts;
        steps += (uint32_t)__popc(reached);
        na += (uint32_t)__popc(accepted);
        if (accepted)
          la = (uint32_t)(kSpecNodes * w) + ((31u - __clz(accepted)) >> 1);
      }
      if (na) {
        curr = share[la / kSpecNodes].L[la % kSpecNodes];
        q = share[la / kSpecNodes].q[la % kSpecNodes];
      }
      if (hit) {
        if (p.eval_trace)
          p.eval_trace[(size_t)s * (C + 1) + ev] = L;
        if (ev > 0 && p.accept_trace)
          p.accept_trace[(size_t)s * C + ev - 1] = (uint8_t)((votes >> lane) & 1u);
      }
      rate = __fdividef(kRateWeight * rate + (float)na,
                        kRateWeight + (float)(steps - (e == 0 ? 1u : 0u)));
      e += steps;
      n_evals += (unsigned)__popc(__ballot_sync(FULL, lead_lane && valid));
      n_acc += na;
      ++n_rounds;
      ++n_warp_rounds;
    }
    if (tl == 0) {
      p.quad_out[s] = q.x;
      p.quad_out[N + s] = q.y;
      p.quad_out[2 * (size_t)N + s] = q.z;
      p.quad_out[3 * (size_t)N + s] = q.w;
      if (p.like_out)
        p.like_out[s] = curr;
      share[0].next = min(N, teams) + atomicAdd(p.counter, 1u);
    }
    meet();
    s = share[0].next;
  }
  if (p.stats && n_warp_rounds && lane == 0) {
    atomicAdd(p.stats, n_evals);
    if (wt == 0) {
      atomicAdd(p.stats + 1, n_rounds);
      atomicAdd(p.stats + 2, n_acc);
    }
    atomicAdd(p.stats + 4, n_warp_rounds);
    atomicAdd(p.stats + 5, 32 * n_warp_rounds);
  }
}

// Dynamic shared memory of a generation kernel with P lanes per sample: one
// staging ring (both directions) per group or warp, the warps' draws, and what
// teams share.
__host__ __device__ constexpr size_t stage_bytes(int P) {
  return sizeof(float4) * (size_t)kWarps * (P < 32 ? 32 / P : 1) * kGroupStrideF4 +
         sizeof(Draw) * (size_t)kWarps * kDraws + (P > 32 ? sizeof(TeamShare) * kWarps : 0);
}

// One chunk per launch (the reference's RunHMMOnDevice granularity).  P lanes
// per sample (P/2 evaluations a round); kSub = 2 normalises every 4 sites
// instead of every 8 (for GLs confident enough that 8-site blocks often leave
// the normalisation range).
template <int P, class E, int kSub = 1>
__global__ void __launch_bounds__(kThreads, kMinBlocks) generation_kernel(const GenParams p) {
  __shared__ float4 s_vq[16];
  if (threadIdx.x < 16 && p.vq_table)
    s_vq[threadIdx.x] = p.vq_table[threadIdx.x];
  __syncthreads();
  if constexpr (P > 32) {
    generation_team<P / 32, E, kSub>(p, s_vq);
  } else {
    const OneChunk src{p};
    generation_body<P, E, OneChunk, kSub>(src, p.counter, p.stats, p.error, s_vq);
  }
}

// Many chunks of uneven size in one persistent launch: one queue over all
// samples of all chunks.
template <int P, class E, int kSub = 1>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    generation_multi_kernel(const MultiParams mp) {
  const ManyChunks src{mp};
  generation_body<P, E, ManyChunks, kSub>(src, mp.counter, mp.stats, mp.error, nullptr);
}

// hmm_work after the generation kernel, over the published final
// quadruples.  Pass 1: a block of two warps per 32 samples of a chunk.  Pass 2:
// one warp per part of a sample (kSampleWords words) samples its sites.
constexpr int kWorkThreads = 32;
constexpr size_t kChainSmem = 2 * sizeof(ChainTiles);  // dynamic: one per recursion

template <class Src>
__device__ __forceinline__ void chains_body(const Src &src) {
  uint32_t c, s0;
  src.locate_block(blockIdx.x, c, s0);
  work_chains(src.chunk(c), s0);
}

template <class Src>
__device__ __forceinline__ void sample_body(const Src &src) {
  __shared__ float4 s_pcr[4];  // the mutation-matrix rows
  __shared__ __align__(16) uint32_t s_u[128];  // a span's uniforms
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t c, s, part;
  src.locate_part(blockIdx.x, c, s, part);
  const GenParams &p = src.chunk(c);
  const uint32_t w_lo = part * kSampleWords, w_hi = min(p.wn, w_lo + kSampleWords);
  if (lane < 4)
    s_pcr[lane] = make_float4(p.pc[4 * lane], p.pc[4 * lane + 1], p.pc[4 * lane + 2],
                              p.pc[4 * lane + 3]);
  __syncwarp();
  const uint32_t N = p.N;
  const uint4 q = make_uint4(p.quad_out[s], p.quad_out[N + s], p.quad_out[2 * (size_t)N + s],
                             p.quad_out[3 * (size_t)N + s]);
  work_sample(p, s_pcr, s, q, lane, s_u, w_lo, w_hi);
}

template <int = 0>
__global__ void __launch_bounds__(kChainThreads, 3) work_chains_kernel(const GenParams p) {
  const OneChunk src{p};
  chains_body(src);
}

template <int = 0>
__global__ void __launch_bounds__(kChainThreads, 3) work_chains_multi_kernel(const MultiParams mp) {
  const ManyChunks src{mp};
  chains_body(src);
}

template <int = 0>
__global__ void __launch_bounds__(kWorkThreads) work_sample_kernel(const GenParams p) {
  const OneChunk src{p};
  sample_body(src);
}

template <int = 0>
__global__ void __launch_bounds__(kWorkThreads) work_sample_multi_kernel(const MultiParams mp) {
  const ManyChunks src{mp};
  sample_body(src);
}

}  // namespace glp
