// glp_join.h -- the product alpha . beta of the two halves of an evaluation,
// rounded to binary32, without the binary64 pipe.
//
// Plain C++ or CUDA: log_dot (glp_kernels.cuh) runs this on the device; the host
// build lets the same code be checked on the CPU (built without contraction of
// products and sums).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define GLP_JOIN_FN __host__ __device__ __forceinline__
#else
#define GLP_JOIN_FN inline
#endif

namespace glp {

GLP_JOIN_FN float join_add(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
GLP_JOIN_FN float join_mul(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
GLP_JOIN_FN uint32_t join_bits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t b;
  memcpy(&b, &x, sizeof(b));
  return b;
#endif
}
GLP_JOIN_FN float join_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float x;
  memcpy(&x, &b, sizeof(x));
  return x;
#endif
}

// a + b = s + err exactly.
GLP_JOIN_FN float two_sum(float a, float b, float &err) {
  const float s = join_add(a, b), t = join_add(s, -a);
  err = join_add(join_add(a, -join_add(s, -t)), join_add(b, -t));
  return s;
}

// x . y of four states that are not negative as m 2^e, m in [1, 2) the mantissa
// that the product has in binary64, rounded to binary32 -- or false, and the caller
// takes the product in binary64.
//
// The four products are exact as a float and an error each, and so are their sums
// (s0, s1, s); c, the eight errors added, is off by less than 2^-45 s: none exceeds
// 2^-24 of what it is the error of, they add up to 3 x 2^-24 s, and each of their
// sums is rounded by 2^-24 of itself.  hi + lo = s + c exactly, and hi is the
// nearest float.  The binary64 sum is within 2^-51 of the product as well, so both
// round to hi unless hi + lo lies that close to the middle of two floats: within
// 2^-21 units of hi's last place, tested with eight times that.  A power of two,
// whose neighbours lie at unequal distances, is left to binary64 too.  Seldom: one
// product in 2^17.  Products outside the range where the errors are floats (a
// blocked pass's never are) and invalid ones give false.
GLP_JOIN_FN bool join_product(float x0, float x1, float x2, float x3, float y0, float y1,
                              float y2, float y3, float &m, int &e) {
  const float p0 = join_mul(x0, y0), p1 = join_mul(x1, y1), p2 = join_mul(x2, y2),
              p3 = join_mul(x3, y3);
  float d0, d1, d2;
  const float s0 = two_sum(p0, p1, d0), s1 = two_sum(p2, p3, d1), s = two_sum(s0, s1, d2);
  const float r0 = join_add(fmaf(x0, y0, -p0), fmaf(x1, y1, -p1));
  const float r1 = join_add(fmaf(x2, y2, -p2), fmaf(x3, y3, -p3));
  const float c = join_add(join_add(d0, d1), join_add(d2, join_add(r0, r1)));
  const float hi = join_add(s, c), lo = join_add(c, -join_add(hi, -s));
  const uint32_t bits = join_bits(hi), top = bits & 0x7f800000u;
  e = (int)(bits >> 23) - 127;
  m = join_float((bits & 0x007fffffu) | 0x3f800000u);
  // (1/2 - 2^-18) units of hi's last place, 2^(e - 23)
  const float most = join_mul(join_float(top), 0x1p-24f - 0x1p-41f);
  return hi >= 0x1p-60f && hi < 0x1p127f && (bits & 0x007fffffu) != 0u && fabsf(lo) < most;
}

}  // namespace glp
