// Activations of the recurrent mixers' gates, in fp32, two numbers at a time: packed arithmetic halves the issue slots that these
// kernels are bound by, and there are no slow paths.  NaN stays NaN.
// The exponential is Cody and Waite's reduction by multiples of ln 2 and a polynomial, kept as 2^n and 2^n p with e^w = 2^n (1 + p), so that
// 1 + e^w and 1 - e^w are rounded once and do not cancel.  Errors against 64 bits (rms, of the value) and those of expf, 1 / (1 + expf), tanhf's
// gelu and sqrtf(-expm1f) in brackets: e^-v 2.8e-8 (4.0e-8); sigmoid of 0.7 to 2 2.2e-8 (3.7e-8), of -2 to -0.7 2.7e-8 (4.6e-8); gelu of the
// same 3.2e-8 (3.6e-8) and 9.4e-8 (2.1e-7); root of 0.01 to 0.3 3.0e-8 (3.2e-8), of 0.7 to 2 2.0e-8 (2.0e-8).  The float32 recurrence of 600
// tokens is 3.90e-7 from 64 bits (3.93e-7).  On ex2.approx with its argument's rounding put back e^-v was 6.4e-8 away, all to one side, and the
// recurrence 3.97e-7; the w2048 design's pass takes 0.3 to 0.4 % longer now (2523 and 2530 us, 2558 and 2567).
#pragma once

#include "f32x2.cuh"

namespace kge {
__device__ __forceinline__ float softplusf_(float v) { return v > 20.f ? v : log1pf(expf(v)); }

__device__ __forceinline__ f2 pk1(float v) { return pk(v, v); }
// e^w = 2^n (1 + p) for |w| <= 88, n in the low bits of both numbers of the result.  n = -127 stands for e^w = 0, from w = -87.7 on.
__device__ __forceinline__ f2 exp_parts2(f2 w, f2& p) {
  const f2 t = fma2(w, pk1(1.44269504f), pk1(12582912.f)), n = add2(t, pk1(-12582912.f));
  // w - n ln 2, ln 2 in a part of 16 bits, whose products with n are exact, and the rest
  f2 h = fma2(n, pk1(-0.693145751953125f), w);
  h = fma2(n, pk1(-1.42860677e-6f), h);
  // e^h = 1 + h + h^2 q(h) for |h| <= ln(2) / 2: least largest error of its degree, 3.1e-9
  f2 q = fma2(h, pk1(0.00138145289f), pk1(0.0083687501f));
  q = fma2(q, h, pk1(0.0416683927f));
  q = fma2(q, h, pk1(0.166665196f));
  q = fma2(q, h, pk1(0.49999994f));
  p = fma2(mul2(q, h), h, h);
  return t;
}
// 2^n, or -2^n, of exp_parts2's result
template <bool NEG = false>
__device__ __forceinline__ f2 exp_scale2(f2 t) {
  float a, b;
  upk(t, a, b);
  const uint32_t one = NEG ? 0xbf800000u : 0x3f800000u;
  return pk(__uint_as_float((__float_as_uint(a) << 23) + one), __uint_as_float((__float_as_uint(b) << 23) + one));
}
__device__ __forceinline__ f2 exp_floor2(f2 w) {               // w >= -88
  float a, b;
  upk(w, a, b);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(-88.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(b) : "f"(-88.f));
  return pk(a, b);
}
// e^w for w <= 88
__device__ __forceinline__ f2 exp2_(f2 w) {
  f2 p;
  const f2 k = exp_scale2(exp_parts2(exp_floor2(w), p));
  return fma2(k, p, k);
}
// 1 / (1 + e^-v): the approximate reciprocal of d, the rounded 1 + e^-v, and a Newton step that knows what d was rounded by.  0 below -87.4
__device__ __forceinline__ f2 sigmoid2(f2 v) {
  float a, b, x, y;
  upk(v, a, b);
  a = -a; b = -b;
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(88.f));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(b) : "f"(88.f));
  f2 p;
  const f2 nk = exp_scale2<true>(exp_parts2(exp_floor2(pk(a, b)), p)), nd = fma2(nk, p, add2(nk, pk1(-1.f)));
  const f2 off = fma2(nk, p, add2(fma2(nd, pk1(-1.f), pk1(-1.f)), nk));      // d - 1 is exact
  upk(nd, a, b);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(-a));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(-b));
  const f2 r = pk(x, y);
  return fma2(fma2(off, r, fma2(nd, r, pk1(1.f))), r, r);
}
// 0.5 v (1 + tanh z) = v sigmoid(2 z)
__device__ __forceinline__ f2 gelu_tanh2(f2 v) {
  const f2 v2 = mul2(v, v);
  return mul2(v, sigmoid2(mul2(v, fma2(v2, pk1(2.f * 0.79788456080286536f * 0.044715f), pk1(2.f * 0.79788456080286536f)))));
}
// sqrt(1 - e^(2 w)), w <= 0; the root by the approximate reciprocal root and a Newton step
__device__ __forceinline__ f2 complement_root2(f2 w) {
  f2 p;
  const f2 nk = exp_scale2<true>(exp_parts2(exp_floor2(add2(w, w)), p)), v = fma2(nk, p, add2(nk, pk1(1.f)));
  float a, b;
  upk(v, a, b);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(1.2e-38f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(b) : "f"(1.2e-38f));
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(b));
  const f2 r = pk(a, b), root = mul2(v, r);
  return fma2(fma2(mul2(root, pk1(-1.f)), root, v), mul2(r, pk1(0.5f)), root);
}
}  // namespace kge
