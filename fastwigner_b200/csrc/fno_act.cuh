// GELU and its derivative for the FNO's kernels, in two forms.
//
// The fused kernels: GELU(x) = x Phi(x) with the lower tail q = Phi(-|x|) = exp(-x^2/2) R(|x|): the
// scaled tail R is a polynomial in t = 1/(1 + 0.28 |x|) (the form of Hastings'
// error-function approximations), fitted here by iteratively reweighted least
// squares to 9e-9 absolute in q.  No branches: about 16 instructions, two of
// them special-function ones, where 0.5 x (1 + erff(x / sqrt 2)) takes both
// branches of erff in a mixed warp (about 45).  Against FP64 on [-8, 8] the
// maximum error is 3.8e-7 and the rms 6.1e-8 (the erff form: 4.5e-7, 6.8e-8).
#pragma once
#include <math.h>
#include <stdint.h>

namespace fw {

// q = Phi(-|x|) and e = exp(-x^2/2)
__device__ __forceinline__ void gauss_tail(float x, float& q, float& e) {
  const float t = __fdividef(1.f, fmaf(fabsf(x), 0.28f, 1.f));
  float p = fmaf(t, -1.058084720e-01f, 3.898751623e-01f);
  p = fmaf(p, t, -2.369956854e-01f);
  p = fmaf(p, t, 2.689122243e-01f);
  p = fmaf(p, t, 6.749581555e-02f);
  p = fmaf(p, t, 1.165209461e-01f);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -0.72134752044448169f * x));
  q = p * t * e;
}
// The erff forms, of the unfused kernels: the training forward pass runs them.
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}
// x Phi(x) = max(x, 0) - |x| q; the clamp keeps an infinite x from 0 * inf
__device__ __forceinline__ float gelu_tail(float x) {
  float q, e;
  gauss_tail(x, q, e);
  return fmaf(-fminf(fabsf(x), 3.4e38f), q, fmaxf(x, 0.f));
}

// two FP32 values in one register pair and the packed operations on them (the
// same roundings as the scalar ones, half the instructions)
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// gelu_tail of two values, operation for operation
__device__ __forceinline__ void gelu2(float& x, float& y) {
  const float ax = fabsf(x), ay = fabsf(y);
  float dx, dy, ex, ey;
  unpack2(fma2(pack2(ax, ay), pack2(0.28f, 0.28f), pack2(1.f, 1.f)), dx, dy);
  const uint64_t t = pack2(__fdividef(1.f, dx), __fdividef(1.f, dy));
  uint64_t p = fma2(t, pack2(-1.058084720e-01f, -1.058084720e-01f), pack2(3.898751623e-01f, 3.898751623e-01f));
  p = fma2(p, t, pack2(-2.369956854e-01f, -2.369956854e-01f));
  p = fma2(p, t, pack2(2.689122243e-01f, 2.689122243e-01f));
  p = fma2(p, t, pack2(6.749581555e-02f, 6.749581555e-02f));
  p = fma2(p, t, pack2(1.165209461e-01f, 1.165209461e-01f));
  const uint64_t v = pack2(x, y);
  unpack2(mul2(mul2(v, pack2(-0.72134752044448169f, -0.72134752044448169f)), v), ex, ey);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(ex));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(ey));
  const uint64_t q = mul2(mul2(p, t), pack2(ex, ey));
  unpack2(fma2(pack2(-fminf(ax, 3.4e38f), -fminf(ay, 3.4e38f)), q, pack2(fmaxf(x, 0.f), fmaxf(y, 0.f))), x, y);
}
__device__ __forceinline__ float gelu_d_tail(float x) {
  float q, e;
  gauss_tail(x, q, e);
  return fmaf(x * 0.39894228040143268f, e, x >= 0.f ? 1.f - q : q);
}

}  // namespace fw
