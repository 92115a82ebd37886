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
// nodes; where z is below -1/2 the two terms cancel, and c enters with its low part.  Beyond, by erfc(x) = t exp(p(t) - x^2),
// t = 1 / (1 + x / 2), x = |z| / sqrt(2) (the form in Numerical Recipes; the coefficients are fitted here), p the least-squares
// polynomial of log(erfcx(x) / t) at Chebyshev nodes for x up to 10, off by 4e-8; the argument's rounding and the fast
// exponential make that 6e-7 of the result at z = -2 and 2e-5 at -12.  Error against 64 bits with an exact exponential and
// quotient, erff's in brackets, root mean square: 2.8e-8 (3.9e-8) for z in [-0.5, 3], 8.0e-8 (8.7e-8) in [-1.25, -1], 1.2e-7
// (3.5e-7) in [-2, -1.75].
// Two values at a time, because the products and sums go two an instruction (fma.rn.f32x2: the same bits as two).
__device__ __forceinline__ float2 ts_fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 ts_gelu2(float2 z) {
  constexpr float C = 0.39894229f, C_LOW = -1.1335170e-08f;
  auto both = [](float v) { return make_float2(v, v); };
  const float2 zero = both(-0.f), s = ts_fma2(z, z, zero), half = ts_fma2(z, both(0.5f), zero);
  float2 r = both(5.00851229e-07f);
  r = ts_fma2(r, s, both(-9.16994031e-06f));
  r = ts_fma2(r, s, both(1.15218179e-04f));
  r = ts_fma2(r, s, both(-1.18725025e-03f));
  r = ts_fma2(r, s, both(9.97354649e-03f));
  r = ts_fma2(r, s, both(-6.64903820e-02f));
  const float2 near = ts_fma2(s, ts_fma2(r, s, both(C)), half);
  const float2 below = ts_fma2(s, ts_fma2(r, s, both(C_LOW)), ts_fma2(s, both(C), half));
  // (x / 2 = |z| / sqrt(8); x^2 = s / 2)
  const float2 t = make_float2(__fdividef(1.f, fmaf(0.35355339f, fabsf(z.x), 1.f)), __fdividef(1.f, fmaf(0.35355339f, fabsf(z.y), 1.f)));
  float2 p = both(-0.177510202f);
  p = ts_fma2(p, t, both(0.746688426f));
  p = ts_fma2(p, t, both(-1.033173919f));
  p = ts_fma2(p, t, both(0.400636137f));
  p = ts_fma2(p, t, both(-0.071767755f));
  p = ts_fma2(p, t, both(0.404021591f));
  p = ts_fma2(p, t, both(0.997049689f));
  p = ts_fma2(p, t, both(-1.265386701f));
  p = ts_fma2(s, both(-0.5f), p);
  const float2 zt = ts_fma2(make_float2(fminf(z.x, 16.f), fminf(z.y, 16.f)), t, zero);    // (16: the exponential is zero there, and z may be infinite)
  const float2 e = make_float2(__expf(p.x), __expf(p.y));
  const float2 w = ts_fma2(ts_fma2(zt, both(0.5f), zero), e, zero), rest = ts_fma2(w, both(-1.f), z);
  auto pick = [](float z, float near, float below, float w, float rest) {
    return fabsf(z) < 1.25f ? (z < -0.5f ? below : near) : (z < 0.f ? w : rest);
  };
  return make_float2(pick(z.x, near.x, below.x, w.x, rest.x), pick(z.y, near.y, below.y, w.y, rest.y));
}
__device__ __forceinline__ float ts_gelu(float z) { return ts_gelu2(make_float2(z, z)).x; }
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
