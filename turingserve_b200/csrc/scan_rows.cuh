// What the token-by-token scans over long portions share (lightning.cu, ssm.cu): half a warp owns one or two state columns,
// its 16 lanes the rows, so the products with the state need no barrier inside a token; two 32-bit operations an instruction
// (fma.rn.f32x2: the same bits as two fmaf); and the sums over the lanes of 16 outputs at once.
//
// The order of a row sum is the same in these kernels and in those for a few tokens, whatever the split of rows over
// threads, so that how a prompt is cut changes no bit: parts of eight rows, each (r0 + r2 + r4 + r6) + (r1 + r3 + r5 + r7) as
// two chains of fmaf, then neighbours, pairs of neighbours and so on (a balanced tree over the parts in row order, absent
// rows zero).
#pragma once

#include "common.cuh"
#include "mma_utils.cuh"

namespace scan {

typedef unsigned long long f2;   // two floats, the lower-numbered row in the lower half

__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(f2 v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// A token's row in shared memory, in pieces of four rows: lane p's rows are 8 p .. 8 p + 7 (ROWS 8) or 16 p .. 16 p + 15, its
// k-th piece lies at piece k * 16 + p, so that the 16 lanes read neighbouring pieces.  Where piece c of the row goes:
template <int ROWS>
__device__ __forceinline__ int piece_at(int c) { return (c % (ROWS / 4)) * 16 + c / (ROWS / 4); }

// A token's operands are loaded while the token before is computed.  The first products of a token and the loads of the next
// are asm volatile, which keeps them in this order: all loads share few scoreboards, so a wait for one token's operands must
// not come right behind the loads of the next.
template <int ROWS>
__device__ __forceinline__ void load_rows(uint32_t row, int p, f2 (&v)[ROWS / 2]) {
#pragma unroll
  for (int k = 0; k < ROWS / 4; ++k)
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[2 * k]), "=l"(v[2 * k + 1]) : "r"(row + 16 * (k * 16 + p)));
}
__device__ __forceinline__ float load_f32(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ float2 load_pair(uint32_t at) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at));
  return v;
}
__device__ __forceinline__ f2 mul2_first(f2 a, f2 b) {
  f2 d;
  asm volatile("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// The products of one state column's rows with q, summed within the lane (`first` starts the first row's chain).  `second`: the
// second part of 16 rows exists.  (Absent rows have keys and queries of zero, but times an infinite value that is NaN: absent
// parts are left out here, and a lane without any row takes its value from a place that holds zero.)
template <int ROWS>
__device__ __forceinline__ float dot_rows(const f2 (&s)[ROWS / 2], const f2 (&q)[ROWS / 2], float first, bool second) {
  float part[ROWS / 8];
#pragma unroll
  for (int m = 0; m < ROWS / 8; ++m) {
    f2 e = pack2(m == 0 ? first : 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) e = fma2(s[4 * m + i], q[4 * m + i], e);
    const float2 v = unpack2(e);
    part[m] = v.x + v.y;
  }
  return ROWS == 8 ? part[0] : part[0] + (second ? part[ROWS / 8 - 1] : 0.f);
}

// x[i] of every lane summed over the 16 lanes of its half warp; lane p gets the sum of x[p].  15 shuffles for 16 sums; lanes
// are joined first with their neighbours (lane ^ 1), last with lane ^ 8.
__device__ __forceinline__ float sum_scatter(float (&x)[16], int lane) {
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const bool up = (lane >> b) & 1;
#pragma unroll
    for (int i = 0; i < (8 >> b); ++i) {
      const float keep = up ? x[2 * i + 1] : x[2 * i], send = up ? x[2 * i] : x[2 * i + 1];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1 << b);
    }
  }
  return x[0];
}

// The sums of `parts` (at most 32) groups of eight rows, `stride` apart, as the tree above.
// FEW: with a way for few parts (planned instances: keys of 64 3 % faster, of 16 12 %; in the lean ones keys of 128 would lose 4 %).
template <int MOST>
__device__ __forceinline__ float tree_of(const float* p, int parts, int stride) {
  float x[MOST];
#pragma unroll
  for (int i = 0; i < MOST; ++i) x[i] = i < parts ? p[i * stride] : 0.f;
#pragma unroll
  for (int n = MOST / 2; n > 0; n >>= 1)
#pragma unroll
    for (int i = 0; i < n; ++i) x[i] = x[2 * i] + x[2 * i + 1];
  return x[0];
}
template <bool FEW>
__device__ __forceinline__ float tree_of_parts(const float* p, int parts, int stride) {
  if (FEW && parts == 16) return tree_of<16>(p, 16, stride);               // (keys of 128 first)
  if (FEW && parts <= 4) return tree_of<4>(p, parts, stride);              // (absent parts add nothing)
  if (FEW && parts <= 8) return tree_of<8>(p, parts, stride);
  const float x = tree_of<16>(p, parts, stride);
  return parts > 16 ? x + tree_of<16>(p + 16 * stride, parts - 16, stride) : x;
}

}  // namespace scan
