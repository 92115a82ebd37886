// One-input activations of the feed-forwards, in 32-bit.
#pragma once

#include "common.cuh"

enum TsActivation : int { TS_ACT_NONE = 0, TS_ACT_GELU_TANH = 1, TS_ACT_RELU2 = 2, TS_ACT_SILU = 3, TS_ACT_GELU = 4 };
constexpr int TS_ACT_LAST = 4;

__device__ __forceinline__ float ts_activate(float z, int kind) {
  if (kind == TS_ACT_GELU_TANH) return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
  if (kind == TS_ACT_RELU2) {
    const float r = fmaxf(z, 0.f);
    return r * r;
  }
  if (kind == TS_ACT_SILU) return z / (1.f + expf(-z));
  if (kind == TS_ACT_GELU) return 0.5f * z * (1.f + erff(0.7071067811865476f * z));
  return z;
}

// The same on its way to a rounding to T: for bfloat16 the tanh form of GELU is z * sigmoid(2 u), u = 0.79788456 (z +
// 0.044715 z^3), with the hardware's approximate exponential and reciprocal (about 2^-21 relative, against a bfloat16 step of
// 2^-9), and SiLU likewise; the error-function form is ts_gelu; the 32-bit type keeps the exact functions.
template <typename T> __device__ __forceinline__ float ts_activate_for(float z, int kind) { return ts_activate(z, kind); }
// z Phi(z) in 32 bits without erff's branches, which cost the epilogue that applies this to a product's tile more than the
// product itself.  |z| < 1.25: z / 2 + s (c + s R(s)), s = z^2, c = 1 / sqrt(2 pi), R the least-squares polynomial at Chebyshev
// nodes; where z is below -1/2 the two terms cancel, and s and c enter with their low parts.  Beyond, by erfc(x) = t exp(p(t) -
// x^2), t = 1 / (1 + x / 2), x = |z| / sqrt(2) (the form in Numerical Recipes; the coefficients are fitted here), p the least-squares polynomial of log(erfcx(x) / t) at
// Chebyshev nodes for x up to 10, off by 4e-8; the argument's rounding and the fast exponential make that 7e-7 of the result at
// z = -2 and 2e-5 at -12.  Against 64 bits, with erff in brackets: root
// mean square 2.8e-8 (3.9e-8) for z in [-0.5, 3], 5.9e-8 (8.7e-8) in [-1.25, -1], 1.8e-7 (3.5e-7) in [-2, -1.75], and nowhere more
__device__ __forceinline__ float ts_gelu(float z) {
  constexpr float C = 0.39894229f, C_LOW = -1.1335170e-08f;
  const float s = z * z, half = 0.5f * z;
  float r = 5.00851229e-07f;
  r = fmaf(r, s, -9.16994031e-06f);
  r = fmaf(r, s, 1.15218179e-04f);
  r = fmaf(r, s, -1.18725025e-03f);
  r = fmaf(r, s, 9.97354649e-03f);
  r = fmaf(r, s, -6.64903820e-02f);
  const float core = z < -0.5f ? fmaf(s, fmaf(r, s, C_LOW), fmaf(fmaf(z, z, -s), C, fmaf(s, C, half))) : fmaf(s, fmaf(r, s, C), half);
  const float x = 0.7071067811865476f * fabsf(z), t = __fdividef(1.f, fmaf(0.5f, x, 1.f));
  float p = -0.177510202f;
  p = fmaf(p, t, 0.746688426f);
  p = fmaf(p, t, -1.033173919f);
  p = fmaf(p, t, 0.400636137f);
  p = fmaf(p, t, -0.071767755f);
  p = fmaf(p, t, 0.404021591f);
  p = fmaf(p, t, 0.997049689f);
  p = fmaf(p, t, -1.265386701f);
  const float e = 0.5f * t * __expf(fmaf(-x, x, p));
  const float tail = z < 0.f ? z * e : fmaf(-fminf(z, 16.f), e, z);       // (16: e is zero there, and z may be infinite)
  return fabsf(z) < 1.25f ? core : tail;
}
template <> __device__ __forceinline__ float ts_activate_for<bf16>(float z, int kind) {
  if (kind == TS_ACT_GELU_TANH) return __fdividef(z, 1.f + __expf(-1.5957691216057308f * (z + 0.044715f * z * z * z)));
  if (kind == TS_ACT_SILU) return __fdividef(z, 1.f + __expf(-z));
  if (kind == TS_ACT_GELU) return ts_gelu(z);
  return ts_activate(z, kind);
}

// A gated unit whose inputs are clamped: g <- min(g, limit), u <- clamp(u, -limit, limit), g sigmoid(slope g) (u + offset).
struct TsGlu {
  float limit, slope, offset;
};
template <typename T> __device__ __forceinline__ float ts_glu_for(float g, float u, const TsGlu& a) {
  g = fminf(g, a.limit);
  u = fminf(fmaxf(u, -a.limit), a.limit);
  return g / (1.f + expf(-a.slope * g)) * (u + a.offset);
}
template <> __device__ __forceinline__ float ts_glu_for<bf16>(float g, float u, const TsGlu& a) {
  g = fminf(g, a.limit);
  u = fminf(fmaxf(u, -a.limit), a.limit);
  return __fdividef(g, 1.f + __expf(-a.slope * g)) * (u + a.offset);
}
