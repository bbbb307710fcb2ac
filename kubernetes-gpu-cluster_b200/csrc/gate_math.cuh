// Activations of the recurrent mixers' gates, in fp32, two numbers at a time: packed arithmetic halves the issue slots that these
// kernels are bound by, and there are no slow paths.  NaN stays NaN.
#pragma once

#include "f32x2.cuh"

namespace kge {
__device__ __forceinline__ float softplusf_(float v) { return v > 20.f ? v : log1pf(expf(v)); }

__device__ __forceinline__ f2 pk1(float v) { return pk(v, v); }
__device__ __forceinline__ f2 clamp2(f2 v, float lo, float hi) {
  float a, b;
  upk(v, a, b);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(lo));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(b) : "f"(lo));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(hi));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(b) : "f"(hi));
  return pk(a, b);
}
// e^-v for |v| < 1e30: 2^(-v log2(e)), the rounding of that product (and of the constant) put back to first order
__device__ __forceinline__ f2 exp_neg2(f2 v) {
  constexpr float L = 1.44269504f, L2 = 1.925963e-8f;          // log2(e) in two parts: 1.44269502162933 + 1.9259630e-8
  const f2 hi = mul2(v, pk1(-L));
  f2 lo = fma2(v, pk1(-L), mul2(v, pk1(L)));
  lo = fma2(v, pk1(-L2), lo);
  float a, b;
  upk(hi, a, b);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b));
  const f2 e = pk(a, b);
  return fma2(e, mul2(lo, pk1(0.693147181f)), e);
}
// 1 / d for 1 <= d < 2^126: the approximate reciprocal and a Newton step
__device__ __forceinline__ f2 recip_from_one2(f2 d) {
  float a, b, x, y;
  upk(d, a, b);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(a));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  const f2 r = pk(x, y);
  return fma2(fma2(mul2(d, pk1(-1.f)), r, pk1(1.f)), r, r);
}
__device__ __forceinline__ f2 sigmoid2(f2 v) { return recip_from_one2(add2(pk1(1.f), exp_neg2(clamp2(v, -87.f, 87.f)))); }      // 1.6e-38 at the lower end
// 0.5 v (1 + tanh z) = v sigmoid(2 z)
__device__ __forceinline__ f2 gelu_tanh2(f2 v) {
  const f2 v2 = mul2(v, v);
  return mul2(v, sigmoid2(mul2(v, fma2(v2, pk1(2.f * 0.79788456080286536f * 0.044715f), pk1(2.f * 0.79788456080286536f)))));
}
// sqrt(1 - e^(-2 x)), x >= 0, a = e^-x: by the power series of 1 - e^-y below y = 1 (its eleventh term is y^11 / 11!, 2.5e-8 of the whole),
// where 1 - a^2 would cancel, and as that above; the root by the approximate reciprocal root and a Newton step
__device__ __forceinline__ f2 complement_root2(f2 x, f2 a) {
  const f2 y = add2(x, x);
  f2 s = pk1(-1.f / 3628800.f);
  s = fma2(s, y, pk1(1.f / 362880.f));
  s = fma2(s, y, pk1(-1.f / 40320.f));
  s = fma2(s, y, pk1(1.f / 5040.f));
  s = fma2(s, y, pk1(-1.f / 720.f));
  s = fma2(s, y, pk1(1.f / 120.f));
  s = fma2(s, y, pk1(-1.f / 24.f));
  s = fma2(s, y, pk1(1.f / 6.f));
  s = fma2(s, y, pk1(-0.5f));
  s = fma2(s, y, pk1(1.f));
  s = mul2(s, y);
  const f2 c = fma2(mul2(a, pk1(-1.f)), a, pk1(1.f));
  float y0, y1, s0, s1, c0, c1, r0, r1;
  upk(y, y0, y1);
  upk(s, s0, s1);
  upk(c, c0, c1);
  const float v0 = y0 < 1.f ? s0 : c0, v1 = y1 < 1.f ? s1 : c1;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r0) : "f"(v0), "f"(1e-30f));
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r1) : "f"(v1), "f"(1e-30f));
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(r0));
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(r1));
  const f2 v = pk(v0, v1), r = pk(r0, r1), root = mul2(v, r);
  return fma2(fma2(mul2(root, pk1(-1.f)), root, v), mul2(r, pk1(0.5f)), root);
}
__device__ __forceinline__ float first2(f2 v) { float a, b; upk(v, a, b); return a; }
}  // namespace kge
