"""The codec's quotients against the compiler's division, bit for bit: random
operands over the range that takes the short form and beyond it, the range's ends,
mantissas of ones and powers of two, zero numerators of both signs."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

SRC = r'''
#include "glp_rng.h"
#include "glp_vq.cuh"
__device__ float pick(uint32_t r, uint32_t kind, int lo, int hi) {
  // kind 0: any mantissa; 1: next to a power of two, or of ones
  const int e = lo + (int)((r >> 23) % (uint32_t)(hi - lo + 1)) + 127;
  uint32_t m = r & 0x7fffffu;
  if (kind)
    m = (m & 4u) ? 0x7fffffu - (m & 3u) : (m & 3u);
  return __uint_as_float((uint32_t)e << 23 | m);
}
__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}
// counts: [0] differing quotients, [1] pairs looked at, [2] of them in the short form
__global__ void quotients(uint64_t seed, uint32_t per, unsigned long long *counts) {
  unsigned long long bad = 0, n = 0, shorts = 0;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  for (uint32_t i = 0; i < per; ++i) {
    const glp_u32x4 x = glp_draw(seed, i, t, 0, 7u), y = glp_draw(seed, i, t, 1, 7u);
    // mostly the range of GLs; else far beyond both ends of the short form's
    const bool far = (y.v[0] & 15u) == 0;
    const float g0 = (y.v[3] & 63u) == 0 ? __uint_as_float(y.v[3] & 0x80000000u)
                                         : pick(x.v[0], y.v[0] >> 30, far ? -126 : -80, far ? 60 : 0);
    const float g1 = pick(x.v[1], (y.v[0] >> 28) & 1u, far ? -126 : -80, far ? 60 : 0);
    const float g2 = pick(x.v[2], (y.v[0] >> 27) & 1u, far ? -60 : -29, far ? 60 : 1);
    const float s = __fadd_rn(__fadd_rn(g0, g1), g2);
    float rr, het;
    glp::vq_normalise(g0, g1, g2, rr, het);
    bad += !same(rr, __fdiv_rn(g0, s)) + !same(het, __fdiv_rn(g1, s));
    shorts += fabsf(s) >= 0x1p-30f && fabsf(s) <= 0x1p30f && glp::vq_quotient_ok(g0) &&
              glp::vq_quotient_ok(g1);
    n += 2;
  }
  atomicAdd(counts, bad);
  atomicAdd(counts + 1, n);
  atomicAdd(counts + 2, 2 * shorts);
}
extern "C" int run(unsigned long long seed, unsigned per, unsigned long long *counts) {
  quotients<<<152 * 8, 256>>>(seed, per, counts);
  return (int)cudaDeviceSynchronize();
}
'''


def test_quotients(tmp_path):
    import torch
    from device_code import compile_launcher
    L = compile_launcher(tmp_path, SRC)
    L.run.argtypes = [C.c_ulonglong, C.c_uint, C.c_void_p]
    counts = torch.zeros(3, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for seed in range(4):
        assert L.run(seed, 1 << 12, counts.data_ptr()) == 0
    bad, n, shorts = counts.tolist()
    assert n == 4 * 152 * 8 * 256 * 2 * (1 << 12)
    assert bad == 0 and 0.5 * n < shorts < 0.99 * n
