"""hmm_work's reciprocals against 1 / x of the compiler, for every float: recip_any
equal everywhere; recip_newton equal from 2^-126 to 2^126, NaN below (subnormal and
zero sums), 0 above and NaN for infinity and NaN -- what its callers test for."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

SRC = r'''
#include "glp_kernels.cuh"
__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}
// counts: [0] recip_any differs, [1] recip_newton differs in its range, [2] outside
// it (both signs), [3] values looked at
__global__ void all_floats(unsigned long long *counts) {
  unsigned long long any = 0, in = 0, out = 0, n = 0;
  for (unsigned long long b = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       b < 1ull << 32; b += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((unsigned)b), want = __frcp_rn(x), a = fabsf(x);
    any += !same(glp::recip_any(x), want);
    const float got = glp::recip_newton(x);
    if (a >= 0x1p-126f && a <= 0x1p126f)
      in += !same(got, want);
    else if (a < 0x1p-126f || a != a || a == __int_as_float(0x7f800000))
      out += got == got;
    else
      out += got != 0.0f;
    ++n;
  }
  atomicAdd(counts, any);
  atomicAdd(counts + 1, in);
  atomicAdd(counts + 2, out);
  atomicAdd(counts + 3, n);
}
extern "C" int run(unsigned long long *counts) {
  all_floats<<<152 * 8, 256>>>(counts);
  return (int)cudaDeviceSynchronize();
}
'''


def test_every_float(tmp_path):
    import torch
    from device_code import compile_launcher
    L = compile_launcher(tmp_path, SRC)
    counts = torch.zeros(4, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert L.run(C.c_void_p(counts.data_ptr())) == 0
    assert counts.tolist() == [0, 0, 0, 2**32]
