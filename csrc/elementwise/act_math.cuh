// Activations of the MLP blocks and their derivatives, for the passes over memory (elementwise.cu) and the GEMM epilogues that
// take their place.
#pragma once
#include "../common/ptx.cuh"

namespace zb {

// erf GELU of two values, x Phi(x), by the tail Q(u) = 1 - Phi(u), u = |x|: with t = 1 / (1 + 0.3 u), exp(u^2 / 2) Q(u) is
// t times a polynomial of degree 7 in t (the form of Abramowitz and Stegun 7.1.26, refitted for the smallest relative
// error, 1.5e-7 over u in [0, 14]).  x Phi(x) = max(x, 0) - u Q(u) then loses nothing in the lower tail, where 1 + erf(x)
// cancels.  Two exponential-unit operations and half of twenty fma slots per value; with erff the passes were bound by
// arithmetic: 3072 x 3072 forward 12.2 us, backward 15.8, now 8.2 and 9.1.  Results that are not the rounded value of 64 bits:
// 171 forward and 153 backward with erff; now, over all normal arguments with normal results, none forward and two backward
// (-4.0e-38 and -1.7e-38, flushed to zero).  The library flushes subnormal numbers: 69 and 7 subnormal results are off.
__device__ __forceinline__ void gelu_tail2(float u0, float u1, float& e0, float& e1, float& q0, float& q1) {
  float d0, d1, s0, s1;
  ffma2(d0, d1, u0, u1, 0.3f, 0.3f, 1.f, 1.f);
  const float t0 = 1.f / d0, t1 = 1.f / d1;
  fmul2(s0, s1, u0, u1, u0, u1);
  fmul2(s0, s1, s0, s1, -0.72134752044448170f, -0.72134752044448170f);   // -u^2 / 2 in powers of two
  e0 = exp2f(s0);
  e1 = exp2f(s1);
  float p0 = 0.03567477688193321f, p1 = p0;
  ffma2(p0, p1, p0, p1, t0, t1, -0.15720310807228088f, -0.15720310807228088f);
  ffma2(p0, p1, p0, p1, t0, t1, 0.20635353028774261f, 0.20635353028774261f);
  ffma2(p0, p1, p0, p1, t0, t1, -0.05368367210030556f, -0.05368367210030556f);
  ffma2(p0, p1, p0, p1, t0, t1, 0.12856164574623108f, 0.12856164574623108f);
  ffma2(p0, p1, p0, p1, t0, t1, 0.09991348534822464f, 0.09991348534822464f);
  ffma2(p0, p1, p0, p1, t0, t1, 0.12075395882129669f, 0.12075395882129669f);
  ffma2(p0, p1, p0, p1, t0, t1, 0.11962930113077164f, 0.11962930113077164f);
  fmul2(p0, p1, p0, p1, t0, t1);
  fmul2(q0, q1, p0, p1, e0, e1);
}
__device__ __forceinline__ float2 gelu_erf_fwd2(float2 x) {
  const float u0 = fabsf(x.x), u1 = fabsf(x.y);
  float e0, e1, q0, q1, r0, r1;
  gelu_tail2(u0, u1, e0, e1, q0, q1);
  fmul2(r0, r1, 0.5f, 0.5f, u0, u1);
  ffma2(r0, r1, 0.5f, 0.5f, x.x, x.y, r0, r1);                            // max(x, 0), a NaN kept
  ffma2(r0, r1, -fminf(u0, 1e30f), -fminf(u1, 1e30f), q0, q1, r0, r1);    // (infinity times the tail's 0 is not wanted)
  return make_float2(r0, r1);
}
// its derivative, Phi(x) + x phi(x)
__device__ __forceinline__ float2 gelu_erf_bwd2(float2 x) {
  float e0, e1, q0, q1, y0, y1;
  gelu_tail2(fabsf(x.x), fabsf(x.y), e0, e1, q0, q1);
  fmul2(y0, y1, x.x, x.y, 0.3989422804014327f, 0.3989422804014327f);
  ffma2(y0, y1, y0, y1, e0, e1, x.x < 0.f ? q0 : 1.f - q0, x.y < 0.f ? q1 : 1.f - q1);
  return make_float2(y0, y1);
}

// kind: 0 = tanh GELU ("gelu_new"), 1 = ReLU; 2 = erf GELU in the forms that take two values
__device__ __forceinline__ float act_fwd(float x, int kind) {
  if (kind == 1) return fmaxf(x, 0.f);
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
}
__device__ __forceinline__ float act_bwd(float x, int kind) {
  if (kind == 1) return x > 0.f ? 1.f : 0.f;
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  float th = tanhf(u);
  return 0.5f * (1.f + th) + 0.5f * x * (1.f - th * th) * k0 * (1.f + 3.f * k1 * x * x);
}
// two values at a time, all kinds
__device__ __forceinline__ float2 act_fwd2(float2 x, int kind) {
  if (kind == 2) return gelu_erf_fwd2(x);
  return make_float2(act_fwd(x.x, kind), act_fwd(x.y, kind));
}
__device__ __forceinline__ float2 act_bwd2(float2 x, int kind) {
  if (kind == 2) return gelu_erf_bwd2(x);
  return make_float2(act_bwd(x.x, kind), act_bwd(x.y, kind));
}

// silu(gate) * up, and the gradients of both
__device__ __forceinline__ float swiglu_fwd(float gate, float up) { return gate / (1.f + __expf(-gate)) * up; }
__device__ __forceinline__ void swiglu_bwd(float gate, float up, float d, float& dgate, float& dup) {
  const float sg = 1.f / (1.f + __expf(-gate));
  const float silu = gate * sg;
  dgate = d * up * (sg * (1.f + gate * (1.f - sg)));
  dup = d * silu;
}

}  // namespace zb
