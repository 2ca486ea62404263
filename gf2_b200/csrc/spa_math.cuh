// Numerics of the flooding sum-product kernel (sm_100a): the operations of
// tanh_half_f and two_atanh_f (numeric.cuh), unrolled for the issue slots.
#pragma once
#include "numeric.cuh"

namespace gf2c {

__device__ __forceinline__ float sf_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// a / b by Markstein's final step (P. Markstein, IBM J. Res. Dev. 34, 1990): with
// y the reciprocal of b (the approximate one and one Newton step) and q = a y, the
// quotient is q + y (a - b q).  It is correctly rounded where y is; one Newton step
// does not promise that of every b, so what is relied on is what was tried on
// sm_100a: each call site below forms both operands from one float, and for every
// value that float can take the result equals __fdiv_rn bit for bit.  A zero keeps
// only its magnitude.
__device__ __forceinline__ float div_cr(float a, float b) {
  float y = sf_rcp(b);
  y = __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
  const float q = __fmul_rn(a, y);
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// tanh(a / 2), a >= 0, and 2 atanh(a), 0 <= a < 1: the operations of tanh_half_f
// and two_atanh_f (numeric.cuh), with selects in place of their branches.
__device__ __forceinline__ float tanh_half_abs(float a) {
  const float inv_ln2 = 1.44269504088896341f;
  const float ln2_hi = 0.693145751953125f;
  const float ln2_lo = 1.42860682030941723e-06f;
  const bool big = a > 30.0f;
  const float x = big ? -30.0f : -a;
  const float kf = rintf(__fmul_rn(x, inv_ln2));
  const float r = __fsub_rn(__fsub_rn(x, __fmul_rn(kf, ln2_hi)), __fmul_rn(kf, ln2_lo));
  float p = 1.0f / 40320.0f;
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 5040.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 720.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 120.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 24.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f / 6.0f);
  p = __fadd_rn(__fmul_rn(p, r), 0.5f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f);
  const float em1r = __fmul_rn(p, r);
  const int k = (int)kf;
  const float two_k = __uint_as_float((uint32_t)(k + 127) << 23);  // k in [-44, 0]
  float em1 = __fadd_rn(__fmul_rn(two_k, em1r), __fsub_rn(two_k, 1.0f));
  em1 = k == 0 ? em1r : em1;
  em1 = big ? -1.0f : em1;
  return div_cr(-em1, __fadd_rn(2.0f, em1));
}
__device__ __forceinline__ float two_atanh_abs(float a) {
  const float y = div_cr(__fmul_rn(2.0f, a), __fsub_rn(1.0f, a));
  const float u = __fadd_rn(1.0f, y);
  // log u
  int e;
  float f = frexp_pos(u, &e);
  const bool low = f < 0.70710678118654752f;
  f = low ? __fmul_rn(f, 2.0f) : f;
  e -= low ? 1 : 0;
  const float g = __fsub_rn(f, 1.0f);
  const float s = __uint_as_float(__float_as_uint(div_cr(fabsf(g), __fadd_rn(f, 1.0f))) ^
                                  (__float_as_uint(g) & 0x80000000u));
  const float s2 = __fmul_rn(s, s);
  float p = 1.0f / 11.0f;
  p = __fadd_rn(__fmul_rn(p, s2), 1.0f / 9.0f);
  p = __fadd_rn(__fmul_rn(p, s2), 1.0f / 7.0f);
  p = __fadd_rn(__fmul_rn(p, s2), 1.0f / 5.0f);
  p = __fadd_rn(__fmul_rn(p, s2), 1.0f / 3.0f);
  p = __fadd_rn(__fmul_rn(p, s2), 1.0f);
  const float lf = __fmul_rn(2.0f, __fmul_rn(s, p));
  const float ln2_hi = 0.693145751953125f;
  const float ln2_lo = 1.42860682030941723e-06f;
  const float ef = (float)e;
  const float l = __fadd_rn(__fadd_rn(__fmul_rn(ef, ln2_hi), lf), __fmul_rn(ef, ln2_lo));
  const bool one = u == 1.0f;
  const float z = __fmul_rn(l, div_cr(y, one ? 1.0f : __fsub_rn(u, 1.0f)));
  return one ? y : z;
}

}  // namespace gf2c
