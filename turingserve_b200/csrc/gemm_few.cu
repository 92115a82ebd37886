// bfloat16 products of a decode step's few tokens (at most 16):
//   out[M, N] = x[M, K] . w[N, K]^T (+ bias[N])          (turingserve/ops/reference.py:45-47)
// The reference leaves them to cuBLAS (turingserve/ops/triton_ops.py:74-76).
//
// A step is a chain of such products, each bound by the weights' bytes or, where those are few, by its latency.  So every
// lane fetches the 16 bytes of weights that it hands to mma.sync (m16n8k16) itself: no layout change, block-wide barrier or
// tensor memory on their way, and none of shared memory either where a warp's share fits its registers (plans 1 and 2; the
// others pass them through a ring of the lane's own).  The first of them are fetched before the wait for the kernel
// before.  The tokens are the product's 16 rows, eight weight rows its columns.  A lane's 16 bytes of weight row
// lane / 4 are eight neighbouring columns of K, which stand for columns 2t, 2t+1, 2t+8, 2t+9 of two products; the
// same permutation on the tokens' side leaves the sum as it is.
//
// Two forms.  few_kernel: the warps of a block cut K between them, a block has one tile of 8 R weight rows, and as every
// token's column is read by one warp only, tokens come from L2 to the warp too (N up to a few thousand).  few_rows_kernel:
// the tokens stand in shared memory and a block of 16 warps an SM takes tiles one after the other (the gate/up product, the
// output head).  What does not fit the registers at once goes through a ring of cp.async copies in which every
// lane has 16 bytes of its own per slot and waits for nobody else.  Sums over K are in the order of the warps, whatever
// finishes the product, so that a product that finishes itself (activation, rotation and cache write, residual add) has
// the bits of the product followed by the kernel that would do it.
#include "activations.cuh"
#include "common.cuh"
#include "mma_utils.cuh"

namespace {

enum FewMode : int { FEW_BF16 = 0, FEW_FLOAT = 1, FEW_GATED = 2, FEW_ROPE = 3, FEW_RESID = 4, FEW_STREAM = 5, FEW_ACT = 6 };

struct FewArgs {
  const bf16* x;          // [M, K]
  const bf16* w;          // [N, K]
  const bf16* bias;       // [N] or null
  void* out;              // [M, N] bf16 / float; [M, N / 2] (gated); the residual rows [M, N], bf16 or 32-bit (added to in place)
  int act;                // FEW_ACT: which activation
  int M, N, K;
  int tiles;              // of 8 R weight rows
  int mode;
  int pairs;              // two neighbouring outputs may be read and written together: N even, out on their boundary
  // FEW_ROPE
  const int* positions;
  const float* cos_t;     // [positions][D / 2]
  const float* sin_t;
  const int* slots;
  bf16* k_cache;
  bf16* v_cache;
  int page, H, KVH, D;
};

__device__ __forceinline__ uint4 ld_weights(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// A lane's own copy to shared memory and the wait for it: no barrier stands between them and the lane's reads, so these
// (unlike cp_async_16 and cp_async_wait) keep the compiler from moving a read across.
__device__ __forceinline__ void own_copy(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
template <int N> __device__ __forceinline__ void own_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Weight row behind column `n` (0..7) of tile `tile`: neighbours, or, where the columns are pairs (gate and up, the two
// halves a rotation joins), columns 2i and 2i + 1 are the two of a pair.
__device__ __forceinline__ int few_row(const FewArgs& a, int tile, int n) {
  int row = tile * 8 + n;
  if (a.mode == FEW_GATED) {
    const int j = tile * 4 + (n >> 1);
    row = (j >> 6) * 128 + (j & 63) + (n & 1) * 64;
  } else if (a.mode == FEW_ROPE) {
    const int half = a.D >> 1, q = tile * 4 + (n >> 1), head = q / half;
    row = head * a.D + (q - head * half) + (n & 1) * half;
  }
  return min(row, a.N - 1);
}

// What finishes two neighbouring columns (pair q = 4 tile + t) of a token: b0, b1 their bias, old the residual's two.
__device__ __forceinline__ void few_finish(const FewArgs& a, int m, int q, float v0, float v1, float b0, float b1, float2 old) {
  if (m >= a.M) return;
  if (a.mode == FEW_GATED) {
    if (2 * q >= a.N) return;
    const float gate = round_to<bf16>(v0), up = round_to<bf16>(v1);
    const float s = round_to<bf16>(silu_for<bf16>(gate));
    reinterpret_cast<bf16*>(a.out)[(size_t)m * (a.N >> 1) + q] = __float2bfloat16_rn(s * up);
    return;
  }
  if (a.mode == FEW_ROPE) {
    const int half = a.D >> 1, head = q / half, p = q - head * half;
    if (head >= a.H + 2 * a.KVH) return;
    const float x1 = round_to<bf16>(v0 + b0), x2 = round_to<bf16>(v1 + b1);
    float o1 = x1, o2 = x2;
    if (head < a.H + a.KVH) {
      const int pos = a.positions[m];
      const float cs = round_to<bf16>(a.cos_t[(size_t)pos * half + p]), sn = round_to<bf16>(a.sin_t[(size_t)pos * half + p]);
      o1 = x1 * cs - x2 * sn;
      o2 = x2 * cs + x1 * sn;
    }
    const bf16 w1 = __float2bfloat16_rn(o1), w2 = __float2bfloat16_rn(o2);
    bf16* qkv = reinterpret_cast<bf16*>(a.out) + (size_t)m * a.N + head * a.D + p;
    qkv[0] = w1;
    qkv[half] = w2;
    if (head >= a.H && a.k_cache != nullptr) {
      const int slot = a.slots[m];
      if (slot >= 0) {
        const bool is_k = head < a.H + a.KVH;
        bf16* dst = (is_k ? a.k_cache : a.v_cache) + ((size_t)(slot / a.page) * a.KVH * a.page + (size_t)(slot % a.page)) * a.D +
                    (size_t)(head - a.H - (is_k ? 0 : a.KVH)) * a.page * a.D;
        dst[p] = w1;
        dst[p + half] = w2;
      }
    }
    return;
  }
  const int n = 2 * q;
  if (n >= a.N) return;
  v0 += b0;
  v1 += b1;
  const size_t at = (size_t)m * a.N + n;
  const bool both = n + 1 < a.N, together = a.pairs;
  if (a.mode == FEW_FLOAT) {
    float* o = reinterpret_cast<float*>(a.out) + at;
    if (together) *reinterpret_cast<float2*>(o) = make_float2(v0, v1);
    else {
      o[0] = v0;
      if (both) o[1] = v1;
    }
    return;
  }
  if (a.mode == FEW_STREAM) {
    float* o = reinterpret_cast<float*>(a.out) + at;
    v0 = old.x + round_to<bf16>(v0);
    v1 = old.y + round_to<bf16>(v1);
    if (together) *reinterpret_cast<float2*>(o) = make_float2(v0, v1);
    else {
      o[0] = v0;
      if (both) o[1] = v1;
    }
    return;
  }
  if (a.mode == FEW_RESID) {
    v0 = round_to<bf16>(v0) + old.x;
    v1 = round_to<bf16>(v1) + old.y;
  } else if (a.mode == FEW_ACT) {
    v0 = ts_activate(round_to<bf16>(v0), a.act);
    v1 = ts_activate(round_to<bf16>(v1), a.act);
  }
  bf16* o = reinterpret_cast<bf16*>(a.out) + at;
  if (together) *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(v0, v1);
  else {
    o[0] = __float2bfloat16_rn(v0);
    if (both) o[1] = __float2bfloat16_rn(v1);
  }
}

// The two columns of a pair in the product's own order.
__device__ __forceinline__ int2 few_columns(const FewArgs& a, int q) {
  if (a.mode != FEW_ROPE) return make_int2(2 * q, 2 * q + 1);
  const int half = a.D >> 1, head = q / half, n0 = head * a.D + (q - head * half);
  return make_int2(n0, n0 + half);
}

__device__ __forceinline__ float2 few_bias(const FewArgs& a, int2 n) {
  float2 b = make_float2(0.f, 0.f);
  if (a.bias == nullptr) return b;
  if (n.x < a.N) b.x = to_f(a.bias[n.x]);
  if (n.y < a.N) b.y = to_f(a.bias[n.y]);
  return b;
}

__device__ __forceinline__ float2 few_old(const FewArgs& a, int m, int q) {
  const int n = 2 * q;
  if ((a.mode != FEW_RESID && a.mode != FEW_STREAM) || m >= a.M || n >= a.N) return make_float2(0.f, 0.f);
  if (a.mode == FEW_STREAM) {
    const float* r = reinterpret_cast<const float*>(a.out) + (size_t)m * a.N + n;
    if (a.pairs) return *reinterpret_cast<const float2*>(r);
    return make_float2(r[0], n + 1 < a.N ? r[1] : 0.f);
  }
  const bf16* r = reinterpret_cast<const bf16*>(a.out) + (size_t)m * a.N + n;
  if (a.pairs) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(r));
  return make_float2(to_f(r[0]), n + 1 < a.N ? to_f(r[1]) : 0.f);
}

// Bias, residual and finish of two columns, out of line: inside the unrolled ring every place would hold a copy of all kinds.
__device__ __noinline__ void few_store(const FewArgs& a, int m, int q, float v0, float v1) {
  const float2 b = few_bias(a, few_columns(a, q));
  few_finish(a, m, q, v0, v1, b.x, b.y, few_old(a, m, q));
}

__host__ __device__ constexpr int few_ldx(int K) { return (K + 31) / 32 * 32 + ((K + 31) / 32 % 2 == 0 ? 32 : 0); }   // (rows an odd number of 64 bytes: no bank conflicts)

// TT: 8 TT tokens at most.  R: tiles of eight weight rows a warp works on at a time.  WK warps cut K.  U: 16-byte loads of
// weights a lane keeps under way, times R; with RING in shared memory.
template <int TT, int R, int WK, int U, bool RING>
__global__ void __launch_bounds__(WK * 32, 1) few_kernel(const __grid_constant__ FewArgs a) {
  pdl_launch_dependents();
  constexpr int ITEMS = R * TT * 32;
  static_assert(ITEMS <= WK * 32, "a thread finishes one pair of columns");
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wk = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int steps = (a.K + 31) >> 5, per = (steps + WK - 1) / WK;
  const int s0 = wk * per, ns = max(0, min(steps, s0 + per) - s0);

  constexpr int SLOT = (R + TT) * 512;
  unsigned char* ring = smem + (size_t)wk * U * SLOT + lane * 16;          // RING: this lane's own 16 bytes of every 512
  uint4 wb[RING ? 1 : U][R], xb[RING ? 1 : U][TT];
  const bf16* wp[R];
#pragma unroll
  for (int r = 0; r < R; ++r) wp[r] = a.w + (size_t)few_row(a, blockIdx.x * R + r, g) * a.K + s0 * 32 + 8 * t;
  auto fetch = [&](int i, int u) {
    if (i < ns) {
      const bool in = (s0 + i) * 32 + 8 * t < a.K;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if constexpr (RING) own_copy(ring + u * SLOT + r * 512, in ? wp[r] + i * 32 : a.w, in);
        else wb[u][r] = in ? ld_weights(wp[r] + i * 32) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  auto fetch_x = [&](int i, int u) {
    if (i < ns) {
      const int k = (s0 + i) * 32 + 8 * t;
#pragma unroll
      for (int h = 0; h < TT; ++h) {
        const bool in = k < a.K && g + 8 * h < a.M;
        const bf16* from = a.x + (in ? (size_t)(g + 8 * h) * a.K + k : 0);
        if constexpr (RING) own_copy(ring + u * SLOT + (R + h) * 512, from, in);
        else xb[u][h] = in ? __ldcg(reinterpret_cast<const uint4*>(from)) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
#pragma unroll
  for (int u = 0; u < U; ++u) fetch(u, u);
  if constexpr (RING) cp_async_commit();
  // the rest of this warp's weights start towards L2
  for (int off = U * 32 + t * 64; off < ns * 32; off += 256)
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (s0 * 32 + 8 * t + off < a.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(wp[r] + off));
  // the two columns that this thread finishes, where the warps' sums meet in shared memory
  const int it = threadIdx.x, i_t = it & 3, i_m = (it >> 2) % (8 * TT), i_r = it / (32 * TT);
  const int i_q = (blockIdx.x * R + i_r) * 4 + i_t;
  float2 old2 = make_float2(0.f, 0.f);
  bf16 bias_x = __ushort_as_bfloat16(0), bias_y = bias_x;
  const int2 i_n = few_columns(a, i_q);
  // (the bias is no part of what may be read early: it starts towards L2 and is read after the wait, behind the tokens, as it is
  // needed last.  Read before the wait it would save a q/k/v product of one token 0.25 us; without the prefetch it costs 0.4)
  if (it < ITEMS && a.bias != nullptr) {
    if (i_n.x < a.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.bias + i_n.x));
    if (i_n.y < a.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.bias + i_n.y));
  }
  pdl_wait();
  if (it < ITEMS) old2 = few_old(a, i_m, i_q);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    fetch_x(u, u);
    if constexpr (RING) cp_async_commit();
  }
  if (it < ITEMS && a.bias != nullptr) {
    if (i_n.x < a.N) bias_x = a.bias[i_n.x];
    if (i_n.y < a.N) bias_y = a.bias[i_n.y];
  }

  float acc[R][2][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[r][0][e] = acc[r][1][e] = 0.f;
  for (int i = 0; i < ns; i += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i + u < ns) {
        constexpr int Z = 0;
        const int o = RING ? Z : u;
        if constexpr (RING) {
          own_wait<U - 1>();
#pragma unroll
          for (int r = 0; r < R; ++r) wb[0][r] = *reinterpret_cast<const uint4*>(ring + u * SLOT + r * 512);
#pragma unroll
          for (int h = 0; h < TT; ++h) xb[0][h] = *reinterpret_cast<const uint4*>(ring + u * SLOT + (R + h) * 512);
        }
        const uint4 x0 = xb[o][0], x1 = TT == 2 ? xb[o][TT - 1] : make_uint4(0u, 0u, 0u, 0u);
        const unsigned a0[4] = {x0.x, x1.x, x0.y, x1.y}, a1[4] = {x0.z, x1.z, x0.w, x1.w};
#pragma unroll
        for (int r = 0; r < R; ++r) {
          mma_bf16(acc[r][0], a0, wb[o][r].x, wb[o][r].y);
          mma_bf16(acc[r][1], a1, wb[o][r].z, wb[o][r].w);
        }
        fetch(i + u + U, u);
        fetch_x(i + u + U, u);
        if constexpr (RING) cp_async_commit();
      }
    }
  }
  // [r][wk][token][4] pairs of columns
  float2* red = reinterpret_cast<float2*>(smem + (RING ? WK * U * SLOT : 0));
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int h = 0; h < TT; ++h)
      red[((r * WK + wk) * TT + h) * 32 + lane] =
          make_float2(acc[r][0][2 * h] + acc[r][1][2 * h], acc[r][0][2 * h + 1] + acc[r][1][2 * h + 1]);
  __syncthreads();
  if (it < ITEMS) {
    const float2* p = red + (size_t)(i_r * WK) * TT * 32 + i_m * 4 + i_t;
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int k = 0; k < WK; ++k) {
      const float2 v = p[k * TT * 32];
      v0 += v.x;
      v1 += v.y;
    }
    few_finish(a, i_m, i_q, v0, v1, to_f(bias_x), to_f(bias_y), old2);
  }
}

// Many rows: the tokens in shared memory, one block of 16 warps an SM (two: where one round each leaves SMs without).  WK warps cut K of a tile of eight weight rows, 16 / WK tiles
// make a round; a block takes rounds blockIdx.x, + gridDim.x, ... while its rings of U copies a lane run on across them.
constexpr int ROWS_WARPS = 16;
constexpr size_t ROWS_ALONE = 116 * 1024;      // no two of such blocks on an SM

template <int TT, int WK, int U, int PER_SM>
__global__ void __launch_bounds__(ROWS_WARPS * 32, PER_SM) few_rows_kernel(const __grid_constant__ FewArgs a) {
  pdl_launch_dependents();
  constexpr int WN = ROWS_WARPS / WK, THREADS = ROWS_WARPS * 32, ITEMS = WN * TT * 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float2 red[WK > 1 ? 2 : 1][WK > 1 ? ROWS_WARPS * TT * 32 : 1];                  // by turns: [wn][wk][token][4] pairs of columns
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, wk = warp % WK, wn = warp / WK;
  const int steps = (a.K + 31) >> 5, per = (steps + WK - 1) / WK;
  const int s0 = wk * per, ns = max(0, min(steps, s0 + per) - s0);
  const int rounds = (a.tiles + WN - 1) / WN;
  const int mine = (int)blockIdx.x < rounds ? (rounds - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int ldx = few_ldx(a.K);
  unsigned char* ring = smem + (size_t)warp * U * 512 + lane * 16;                           // this lane's own 16 bytes of every 512
  bf16* xs = reinterpret_cast<bf16*>(smem + (size_t)ROWS_WARPS * U * 512);

  // (a tile past the last is the last again, and finishes nothing)
  auto row_at = [&](int round) { return a.w + (size_t)few_row(a, min(round * WN + wn, a.tiles - 1), g) * a.K + s0 * 32 + 8 * t; };
  int l_round = blockIdx.x, l_step = 0, l_left = mine * ns, l_slot = 0;
  const bf16* wp = row_at(l_round);
  auto fetch = [&] {
    if (l_left > 0) {
      const bool in = (s0 + l_step) * 32 + 8 * t < a.K;
      own_copy(ring + l_slot * 512, in ? wp + l_step * 32 : a.w, in);
      --l_left;
      if (++l_step == ns) {
        l_step = 0;
        l_round += gridDim.x;
        if (l_left > 0) wp = row_at(l_round);
      }
    }
    cp_async_commit();
    l_slot = l_slot + 1 == U ? 0 : l_slot + 1;
  };
  for (int u = 0; u < U; ++u) fetch();
  pdl_wait();
  {
    const int chunks = ldx / 8;
    for (int i = threadIdx.x; i < TT * 8 * chunks; i += THREADS) {
      const int m = i / chunks, c = i - m * chunks;
      const bool in = m < a.M && c * 8 < a.K;
      *reinterpret_cast<uint4*>(xs + (size_t)m * ldx + c * 8) =
          in ? __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)m * a.K + c * 8)) : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncthreads();

  const bf16* xrow = xs + (size_t)g * ldx + s0 * 32 + 8 * t;
  int slot = 0;
  for (int k = 0; k < mine; ++k) {
    const int round = blockIdx.x + k * gridDim.x;
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 4
    for (int i = 0; i < ns; ++i) {
      own_wait<U - 1>();
      const uint4 w = *reinterpret_cast<const uint4*>(ring + slot * 512);
      const uint4 x0 = *reinterpret_cast<const uint4*>(xrow + i * 32);
      const uint4 x1 = TT == 2 ? *reinterpret_cast<const uint4*>(xrow + 8 * ldx + i * 32) : make_uint4(0u, 0u, 0u, 0u);
      const unsigned a0[4] = {x0.x, x1.x, x0.y, x1.y}, a1[4] = {x0.z, x1.z, x0.w, x1.w};
      mma_bf16(acc[0], a0, w.x, w.y);
      mma_bf16(acc[1], a1, w.z, w.w);
      fetch();
      slot = slot + 1 == U ? 0 : slot + 1;
    }
    if constexpr (WK == 1) {
      const int q = (round * WN + wn) * 4 + t;
      if (round * WN + wn < a.tiles) {
        few_store(a, g, q, acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]);
        if constexpr (TT == 2) few_store(a, g + 8, q, acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
      }
    } else {
#pragma unroll
      for (int h = 0; h < TT; ++h)
        red[k & 1][(warp * TT + h) * 32 + lane] = make_float2(acc[0][2 * h] + acc[1][2 * h], acc[0][2 * h + 1] + acc[1][2 * h + 1]);
      __syncthreads();
      if ((int)threadIdx.x < ITEMS) {
        const int i_n = threadIdx.x / (TT * 32), at = threadIdx.x % (TT * 32);                // (the first warps finish; one barrier a round)
        const float2* p = red[k & 1] + (size_t)i_n * WK * TT * 32 + at;
        float v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int j = 0; j < WK; ++j) {
          const float2 v = p[j * TT * 32];
          v0 += v.x;
          v1 += v.y;
        }
        if (round * WN + i_n < a.tiles) few_store(a, at >> 2, (round * WN + i_n) * 4 + (at & 3), v0, v1);
      }
    }
  }
  cp_async_wait<0>();
}

template <typename K> int allow_smem(K kernel, size_t smem, size_t* allowed) {
  if (smem <= *allowed) return 0;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    TS_REFUSE((int)e, "ts_linear_few: shared memory %zu: %s", smem, cudaGetErrorString(e));
  }
  *allowed = smem;
  return 0;
}

template <int TT, int R, int WK, int U, bool RING = false>
int launch(FewArgs& a, cudaStream_t s) {
  a.tiles = ceil_div(a.N, 8 * R);
  constexpr size_t smem = (RING ? (size_t)WK * U * (R + TT) * 512 : 0) + (size_t)R * WK * TT * 32 * 8;
  static size_t allowed = 48 * 1024;
  const int rc = allow_smem(few_kernel<TT, R, WK, U, RING>, smem, &allowed);
  if (rc != 0) return rc;
  ts_launch(few_kernel<TT, R, WK, U, RING>, dim3(a.tiles), dim3(WK * 32), smem, s, a);
  TS_LAUNCH_CHECK();
}

template <int TT, int WK, bool TWO = false> int launch_rows(FewArgs& a, cudaStream_t s) {
  constexpr int U = TT == 1 && !TWO ? 12 : (TT == 2 && TWO ? 6 : 8);
  auto kernel = few_rows_kernel<TT, WK, U, TWO ? 2 : 1>;
  a.tiles = ceil_div(a.N, 8);
  size_t smem = (size_t)ROWS_WARPS * U * 512 + (size_t)TT * 8 * few_ldx(a.K) * 2;
  if (smem > 210 * 1024) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_linear_few: %zu bytes of shared memory", smem);
  // (launched while the kernel before still holds some SMs, two blocks would land on those that are free and stay there: an
  // output head of 151,936 x 1,536 took 114 us as a step's last link, 82 with one an SM)
  if (!TWO && smem < ROWS_ALONE) smem = ROWS_ALONE;
  static size_t allowed = 48 * 1024;
  const int rc = allow_smem(kernel, smem, &allowed);
  if (rc != 0) return rc;
  const int rounds = ceil_div(a.tiles, ROWS_WARPS / WK), most = (TWO ? 2 : 1) * ts_sm_count();
  ts_launch(kernel, dim3(rounds < most ? rounds : most), dim3(ROWS_WARPS * 32), smem, s, a);
  TS_LAUNCH_CHECK();
}

// The instances by number (tests ask for one; callers leave it to few_plan).
template <int TT> int launch_plan(FewArgs& a, int plan, cudaStream_t s) {
  switch (plan) {
    case 1: return launch<TT, 2, 16, 3>(a, s);
    case 2: return launch<TT, 2, 8, TT == 1 ? 6 : 4>(a, s);
    case 3: return launch<TT, 2, 16, 6, true>(a, s);
    case 4: return launch<TT, 2, 8, TT == 1 ? 8 : 5, true>(a, s);
    case 5: return launch_rows<TT, 8>(a, s);
    case 6: return launch_rows<TT, 4>(a, s);
    case 7: return launch_rows<TT, 2>(a, s);
    case 8: return launch_rows<TT, 1>(a, s);
    case 9: return launch_rows<TT, 4, true>(a, s);
  }
  TS_REFUSE(TS_ERR_SHAPE, "ts_linear_few: no plan %d", plan);
}

// Which instance, by the sizes alone (so a product's bits do not depend on what finishes it).  Times of a product
// with residual add at 8 tokens, weights from DRAM, in us, against the tcgen05 kernel's:
//  * tiles of 16 rows for at most one block an SM: 16 warps cut K; all of a warp's weights in registers at once while
//    they are few (1,536 x 1,536: 2.3 / 4.6; 2,048 x 1,536: 2.6 / 5.0), else a ring in shared memory (896 x 4,864:
//    3.7 / 5.2; 1,536 x 8,960: 7.3 / 9.2; registers 10.8 there: their waits share six scoreboards).  Very long rows have the
//    bytes to keep tcgen05's bulk copies busy (16 tokens: 1,536 x 18,432 16.9 / 15.7; with the norm behind, 1,536 x 28,416
//    26.6 / 24.2, 256 x 20,480 14.9 / 14.3);
//  * for two blocks an SM: the same with 8 warps (4,632 x 1,536: 4.1 / 6.7; 3,584 x 3,584: 6.4 / 9.3).  Where K is long too,
//    blocks of one tile no longer divide the chip evenly: 3,584 x 18,944 33 / 30, left to tcgen05, and sooner where few SMs
//    have a second block (12 tokens: 2,432 x 8,192 13.4 / 12.0; with the norm, 2,816 x 7,168 13.5 / 12.4, but 2,560 x 7,168
//    13.6 / 14.1);
//  * up to two and a half blocks an SM: still that, while a third round costs less than the rows' kernel below (one token, with the
//    norm: 5,120 x 2,560 9.6 / 9.4, 10.9 by rows; q/k/v 5,120 x 2,304 8.4 / 8.4, 9.1 by rows; 9 tokens, 5,120 x 1,536 8.7 / 8.6,
//    9.9 by rows); above, tcgen05 (5,120 x 4,352 14.0 / 12.4, 5,120 x 5,120 15.2 / 14.0), and up to two and
//    three quarters once K is long (without a norm, 6,144 x 7,168 19.7 / 18.8, 6,144 x 8,192 23.6 / 20.9);
//  * more rows: tokens in shared memory.  Few columns: two blocks of 16 warps an SM, 4 warps a tile (9,728 x 896 5.8 / 6.9, 8,192
//    x 1,536 7.1 / 8.8, 20,480 x 1,024 10.8 / 15.5).  Else one block an SM, 1, 2, 4 or 8 warps a tile, whichever deals the tiles
//    out most evenly (17,920 x 1,536 gated, 1 warp: 11.6 / 12.6; 151,936 x 1,536, 1 and 2 warps: 79 and 78 / 86; 13,440 x 1,536, 1, 2
//    and 4 warps: 10.4, 11.3 and 11.3 / 11.1; 37,888 x 3,584 48 / 54).  Long rows of tokens leave too little room: 6,144 x 3,584
//    12.2 by the second rule, 12.6 by tcgen05; 9 to 16 tokens, 6,144 x 2,304 11.9 / 10.0, 12,288 x 1,536 12.0 / 11.2.
// Clusters that share K further (1,536 x 8,960 over 3 blocks each) lose: 10.5 us against 7.0.
int few_plan(int M, int N, int K) {
  const int tiles16 = ceil_div(N, 16), sms = ts_sm_count();
  if (tiles16 <= sms) return K <= 2048 ? 1 : (K <= (M > 8 ? 16384 : 18432) ? 3 : 0);
  if (tiles16 <= 2 * sms) {
    if (4 * tiles16 < 5 * sms && K > (8 * tiles16 <= 9 * sms ? (M > 8 ? 7168 : 8192) : (M > 8 ? 5120 : 7168))) return 0;
    return K <= 1536 ? 2 : (K <= 8192 ? 4 : 0);
  }
  if (2 * tiles16 <= 5 * sms && K > 1100) {
    if (K <= (M > 8 ? 1900 : 3584)) return 4;
    return 0;
  }
  if (4 * tiles16 <= 11 * sms && K > 6144) return 0;
  if (M > 8 && tiles16 <= 7 * sms && (K > 1900 || tiles16 > 5 * sms)) return 0;
  if (K > 2560 && tiles16 <= 6 * sms) return K <= 8192 ? 4 : 0;
  if (few_ldx(K) > 4600) return 0;                 // (16 tokens and the ring: 220 KB)
  if (few_ldx(K) <= 1600 && (tiles16 <= 5 * sms || K <= 1100)) return 9;
  // rounds of the busiest SM x (four times the steps of a round + what its end costs)
  const int tiles = ceil_div(N, 8), steps = ceil_div(K, 32);
  int best = 0, best_cost = 0;
  for (int wk = 1, plan = 8; wk <= 8; wk *= 2, --plan) {
    const int end = wk == 1 ? 8 : (wk == 2 ? 9 : 5 * wk);
    const int cost = ceil_div(ceil_div(tiles, ROWS_WARPS / wk), sms) * (4 * ceil_div(steps, wk) + end);
    if (best == 0 || cost < best_cost) best = plan, best_cost = cost;
  }
  return best;
}

int run(FewArgs& a, int plan, cudaStream_t s) {
  if (a.M > 16 || a.K % 8 != 0 || a.K <= 0)
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_linear_few: M=%d N=%d K=%d is not taken by this kernel", a.M, a.N, a.K);
  if (((uintptr_t)a.x | (uintptr_t)a.w) & 15) TS_REFUSE(TS_ERR_ALIGN, "ts_linear_few: operands must be 16-byte aligned");
  a.pairs = a.N % 2 == 0 && ((uintptr_t)a.out & (a.mode == FEW_FLOAT || a.mode == FEW_STREAM ? 7 : 3)) == 0;
  if (plan == 0) {
    plan = few_plan(a.M, a.N, a.K);
    if (plan == 0) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_linear_few: N=%d K=%d is faster on tcgen05", a.N, a.K);
  }
  return a.M <= 8 ? launch_plan<1>(a, plan, s) : launch_plan<2>(a, plan, s);
}

}  // namespace

// At most 16 tokens, K a multiple of 8, operands on 16-byte boundaries.  kind: 0 out is bfloat16, 1 float32,
// 2 out[M, N / 2] = silu(g) * u (rows of w in blocks of 64 gates and their 64 ups, N a multiple of 128, no bias),
// 4 out[M, N] += the product, both rounded to bfloat16, 5 the same for 32-bit rows (the product rounded to bfloat16),
// 6 out = act(product rounded to bfloat16), `act` as ts_activation's kind.  plan: 0 = by the sizes (TS_ERR_UNSUPPORTED where
// the tcgen05 kernel is the faster one).
TS_API int ts_linear_few(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int kind, int act,
                         int plan, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (kind < 0 || kind > 6 || kind == FEW_ROPE) TS_REFUSE(TS_ERR_SHAPE, "ts_linear_few: no kind %d", kind);
  if (kind == FEW_GATED && (N % 128 != 0 || bias != nullptr))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_linear_few: gated N=%d is not taken by this kernel", N);
  if (kind == FEW_ACT && (act < 1 || act > TS_ACT_LAST)) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_linear_few: activation %d", act);
  FewArgs a = {};
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.bias = (const bf16*)bias; a.out = out;
  a.M = M; a.N = N; a.K = K;
  a.mode = kind; a.act = act;
  return run(a, plan, (cudaStream_t)stream);
}

// The q/k/v product of at most 16 tokens that rotates and writes the cache itself: arguments as ts_linear_tc_qkv_rope.
TS_API int ts_linear_few_qkv_rope(void* qkv, const void* x, const void* w, const void* bias, const int* positions,
                                  const float* cos_t, const float* sin_t, const int* slots, void* k_cache, void* v_cache, int M,
                                  int H, int KVH, int D, int page, int K, int plan, void* stream) {
  if (M <= 0) return 0;
  if (H <= 0 || KVH <= 0 || (D != 64 && D != 128))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_linear_few_qkv_rope: heads %d, %d of %d are not taken by this kernel", H, KVH, D);
  if (positions == nullptr || cos_t == nullptr || sin_t == nullptr)
    TS_REFUSE(TS_ERR_SHAPE, "ts_linear_few_qkv_rope: positions and tables are needed");
  if (k_cache != nullptr && (v_cache == nullptr || slots == nullptr || page <= 0))
    TS_REFUSE(TS_ERR_SHAPE, "ts_linear_few_qkv_rope: the cache write needs both caches, slots and the page size");
  FewArgs a = {};
  a.x = (const bf16*)x; a.w = (const bf16*)w; a.bias = (const bf16*)bias; a.out = qkv;
  a.M = M; a.N = (H + 2 * KVH) * D; a.K = K;
  a.mode = FEW_ROPE;
  a.positions = positions; a.cos_t = cos_t; a.sin_t = sin_t; a.slots = slots;
  a.k_cache = (bf16*)k_cache; a.v_cache = (bf16*)v_cache;
  a.page = page; a.H = H; a.KVH = KVH; a.D = D;
  return run(a, plan, (cudaStream_t)stream);
}
