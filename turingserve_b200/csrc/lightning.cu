// Linear attention with a per-head decay ("lightning attention"): for every request and head a matrix
// state S [D, V] in 32-bit that lives in a state slot between steps,
//     S_t = lam_h S_{t-1} + k_t v_t^T,     o_t = S_t^T q_t,
// with q, k, v = act(projection) taken from one fused projection row [q (H D) | k (H D) | v (H V) | ...].
// The activation (SiLU) is applied here, rounded to the storage type as the projection's own epilogue
// would round it; everything from there on (products with the state, decay, the state itself, the
// output) is 32-bit.  Output: 32-bit rows [T, H V] (a norm over all heads follows in another kernel).
//
// ts_lightning runs the tokens of a step in order, exactly as written above, for single tokens and for
// portions alike, so how a prompt is cut never changes a bit.  The columns of S are independent of one
// another: one block owns LT_COLS columns of one (head, request) and keeps them in REGISTERS over all tokens
// of the step: thread (part, col) holds rows part * LT_ROWS .. of column col.  Tokens arrive in groups of
// LT_GROUP rows: the raw projection rows of the NEXT group are on their way (cp.async, 16 bytes a copy) while
// the present group is computed; a group is activated out of the raw buffer into 32-bit shared memory; its
// partial outputs of the row parts are summed through shared memory, in part order.  Per token a thread does
// 3 * LT_ROWS 32-bit operations on registers with broadcast loads from shared memory.
#include "common.cuh"
#include "mma_utils.cuh"
#include "scan_rows.cuh"

namespace {

constexpr int LT_GROUP = 16;     // tokens staged at a time
constexpr int LT_COLS = 16;      // state columns per block (half a warp: a warp holds two row parts)
constexpr int LT_ROWS = 8;       // state rows per thread (registers)

template <typename T> __device__ __forceinline__ float act_silu(float z) { return round_to<T>(silu_for<T>(z)); }

// PLAN: an instance of its own for portions (its per-thread plan of copies and activations costs 60 registers more, which
// halves the threads an SM holds: see ts_lightning_ex for where it pays)
template <typename T, bool PLAN>
__global__ void __launch_bounds__(512)
lightning_kernel(float* __restrict__ out, const T* __restrict__ proj, int proj_stride, float* __restrict__ state,
                 const float* __restrict__ decay, const int* __restrict__ q_start, const int* __restrict__ slots,
                 int H, int D, int V, int parts, int fast_rows) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  const int h = blockIdx.y, b = blockIdx.z;
  const int t0 = q_start[b], n = q_start[b + 1] - t0;
  if (n <= 0) return;
  const int Dp = parts * LT_ROWS;                          // D rounded up: rows beyond D hold zero keys and queries
  const int col = threadIdx.x & (LT_COLS - 1), part = threadIdx.x / LT_COLS;
  const int j = blockIdx.x * LT_COLS + col;
  const bool live = j < V;
  const float lam = decay[h];
  float* S = state + ((size_t)slots[b] * H + h) * D * V;
  float* q_s = smem;                                       // [LT_GROUP][Dp]
  float* k_s = q_s + LT_GROUP * Dp;                        // [LT_GROUP][Dp]
  float* v_s = k_s + LT_GROUP * Dp;                        // [LT_GROUP][LT_COLS]
  float* o_s = v_s + LT_GROUP * LT_COLS;                   // [LT_GROUP][parts][LT_COLS]

  float s[LT_ROWS];
#pragma unroll
  for (int i = 0; i < LT_ROWS; ++i) {
    const int d = part * LT_ROWS + i;
    s[i] = (live && d < D) ? S[(size_t)d * V + j] : 0.f;
  }
  const int q_off = h * D, k_off = H * D + h * D, v_off = 2 * H * D + h * V;
  // raw rows of a group, as stored: [2 buffers][LT_GROUP][D q | D k | LT_COLS v] (fast_rows: D a multiple of 8 and
  // every piece 16-byte aligned, so the copies are asynchronous 16-byte ones; else plain loads at activation)
  T* raw = reinterpret_cast<T*>(o_s + LT_GROUP * parts * LT_COLS);
  const int raw_row = 2 * D + LT_COLS;
  const int cols_here = min(LT_COLS, V - (int)blockIdx.x * LT_COLS);
  constexpr int PER16 = 16 / (int)sizeof(T);
  // Which pieces of a group a thread copies, and which it activates, is the same for every group: with PLAN both are
  // worked out once instead of by two divisions a piece and group.  At most LT_MAX_COPIES 16-byte copies a thread (16 rows
  // of 2 D / PER16 + LT_COLS / PER16 pieces over 2 D threads) and LT_MAX_ACT pieces to activate.
  constexpr int LT_MAX_COPIES = 8, LT_MAX_ACT = 4;
  int cp_row[LT_MAX_COPIES], cp_src[LT_MAX_COPIES], cp_dst[LT_MAX_COPIES];
  int ac_row[LT_MAX_ACT], ac_src[LT_MAX_ACT], ac_dst[LT_MAX_ACT];
  const bool planned = PLAN && fast_rows;
  if (planned) {
    const int chunks_qk = D / PER16, chunks_v = LT_COLS / PER16, per_row = 2 * chunks_qk + chunks_v;
#pragma unroll
    for (int k = 0; k < LT_MAX_COPIES; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      cp_row[k] = LT_GROUP;                                // (beyond every group: never copied)
      cp_src[k] = cp_dst[k] = 0;
      if (i < LT_GROUP * per_row) {
        const int r = i / per_row, c = i % per_row;
        if (c < chunks_qk) {
          cp_row[k] = r;
          cp_src[k] = r * proj_stride + q_off + c * PER16;
          cp_dst[k] = r * raw_row + c * PER16;
        } else if (c < 2 * chunks_qk) {
          cp_row[k] = r;
          cp_src[k] = r * proj_stride + k_off + (c - chunks_qk) * PER16;
          cp_dst[k] = r * raw_row + D + (c - chunks_qk) * PER16;
        } else if ((c - 2 * chunks_qk) * PER16 < cols_here) {
          cp_row[k] = r;
          cp_src[k] = r * proj_stride + v_off + blockIdx.x * LT_COLS + (c - 2 * chunks_qk) * PER16;
          cp_dst[k] = r * raw_row + 2 * D + (c - 2 * chunks_qk) * PER16;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < LT_MAX_ACT; ++k) {
      const int i = threadIdx.x + k * blockDim.x;
      ac_row[k] = LT_GROUP;
      ac_src[k] = ac_dst[k] = 0;
      if (i < LT_GROUP * 2 * chunks_qk) {
        const int r = i / (2 * chunks_qk), c = i % (2 * chunks_qk);
        const int which = c >= chunks_qk, cc = (which ? c - chunks_qk : c) * PER16;
        ac_row[k] = r;
        ac_src[k] = r * raw_row + which * D + cc;
        ac_dst[k] = which * LT_GROUP * Dp + r * Dp + cc;   // (k_s lies LT_GROUP * Dp behind q_s)
      }
    }
  }
  auto fetch = [&](int g0, int buf) {
    if (!fast_rows) return;
    if (planned) {
      const int gn = min(LT_GROUP, n - g0);
      const T* first = proj + (size_t)(t0 + g0) * proj_stride;
      T* dst0 = raw + (size_t)buf * LT_GROUP * raw_row;
#pragma unroll
      for (int k = 0; k < LT_MAX_COPIES; ++k)
        if (cp_row[k] < gn) cp_async_16(dst0 + cp_dst[k], first + cp_src[k], true);
      return;
    }
    const int gn = min(LT_GROUP, n - g0);
    const int chunks_qk = D / PER16, chunks_v = LT_COLS / PER16, per_row = 2 * chunks_qk + chunks_v;
    for (int i = threadIdx.x; i < gn * per_row; i += blockDim.x) {
      const int r = i / per_row, c = i % per_row;
      const T* row = proj + (size_t)(t0 + g0 + r) * proj_stride;
      T* dst = raw + ((size_t)buf * LT_GROUP + r) * raw_row;
      if (c < chunks_qk) cp_async_16(dst + c * PER16, row + q_off + c * PER16, true);
      else if (c < 2 * chunks_qk) cp_async_16(dst + D + (c - chunks_qk) * PER16, row + k_off + (c - chunks_qk) * PER16, true);
      else {
        const int cc = (c - 2 * chunks_qk) * PER16;
        const bool ok = cc < cols_here;
        cp_async_16(dst + 2 * D + cc, ok ? row + v_off + blockIdx.x * LT_COLS + cc : proj, ok);
      }
    }
  };
  for (int i = threadIdx.x; i < 2 * LT_GROUP * Dp; i += blockDim.x) q_s[i] = 0.f;      // (q_s and k_s: rows beyond D stay zero)
  fetch(0, 0);
  cp_async_commit();
  int buf = 0;
  for (int g0 = 0; g0 < n; g0 += LT_GROUP, buf ^= 1) {
    const int gn = min(LT_GROUP, n - g0);
    if (g0 + LT_GROUP < n) fetch(g0 + LT_GROUP, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();                                       // this group's raw rows are here; the group before is stored
    if (planned) {
      const T* raw0 = raw + (size_t)buf * LT_GROUP * raw_row;
#pragma unroll
      for (int k = 0; k < LT_MAX_ACT; ++k) {
        if (ac_row[k] < gn) {
          const uint4 rawv = *reinterpret_cast<const uint4*>(raw0 + ac_src[k]);
          const T* e = reinterpret_cast<const T*>(&rawv);
          float* dst = q_s + ac_dst[k];
#pragma unroll
          for (int u = 0; u < PER16; ++u) dst[u] = act_silu<T>(to_f(e[u]));
        }
      }
    } else if (fast_rows) {
      // 16 bytes (PER16 values) of q or k at a time: the index arithmetic once a piece, not once a value
      const int chunks = D / PER16;
      for (int i = threadIdx.x; i < gn * 2 * chunks; i += blockDim.x) {
        const int r = i / (2 * chunks), c = i % (2 * chunks);
        const int which = c >= chunks, cc = (which ? c - chunks : c) * PER16;
        const uint4 rawv = *reinterpret_cast<const uint4*>(raw + ((size_t)buf * LT_GROUP + r) * raw_row + which * D + cc);
        const T* e = reinterpret_cast<const T*>(&rawv);
        float* dst = (which ? k_s : q_s) + r * Dp + cc;
#pragma unroll
        for (int u = 0; u < PER16; ++u) dst[u] = act_silu<T>(to_f(e[u]));
      }
    } else {
      for (int i = threadIdx.x; i < gn * D; i += blockDim.x) {
        const int r = i / D, d = i % D;
        const T* row = proj + (size_t)(t0 + g0 + r) * proj_stride;
        q_s[r * Dp + d] = act_silu<T>(to_f(row[q_off + d]));
        k_s[r * Dp + d] = act_silu<T>(to_f(row[k_off + d]));
      }
    }
    for (int i = threadIdx.x; i < gn * LT_COLS; i += blockDim.x) {
      const int r = i / LT_COLS, c = i % LT_COLS;
      float vv = 0.f;
      if (c < cols_here) {
        vv = fast_rows ? to_f(raw[((size_t)buf * LT_GROUP + r) * raw_row + 2 * D + c])
                       : to_f(proj[(size_t)(t0 + g0 + r) * proj_stride + v_off + blockIdx.x * LT_COLS + c]);
        vv = act_silu<T>(vv);
      }
      v_s[i] = vv;
    }
    __syncthreads();
#pragma unroll 2
    for (int r = 0; r < gn; ++r) {
      const float vj = v_s[r * LT_COLS + col];
      const float4* qr = reinterpret_cast<const float4*>(q_s + r * Dp + part * LT_ROWS);
      const float4* kr = reinterpret_cast<const float4*>(k_s + r * Dp + part * LT_ROWS);
      float o = 0.f, o2 = 0.f;                                 // two chains: the order of scan_rows.cuh
#pragma unroll
      for (int i = 0; i < LT_ROWS / 4; ++i) {
        const float4 k4 = kr[i], q4 = qr[i];
        s[4 * i + 0] = fmaf(lam, s[4 * i + 0], k4.x * vj);
        o = fmaf(s[4 * i + 0], q4.x, o);
        s[4 * i + 1] = fmaf(lam, s[4 * i + 1], k4.y * vj);
        o2 = fmaf(s[4 * i + 1], q4.y, o2);
        s[4 * i + 2] = fmaf(lam, s[4 * i + 2], k4.z * vj);
        o = fmaf(s[4 * i + 2], q4.z, o);
        s[4 * i + 3] = fmaf(lam, s[4 * i + 3], k4.w * vj);
        o2 = fmaf(s[4 * i + 3], q4.w, o2);
      }
      o_s[(r * parts + part) * LT_COLS + col] = o + o2;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < gn * LT_COLS; i += blockDim.x) {
      const int r = i / LT_COLS, c = i % LT_COLS;
      const int jj = blockIdx.x * LT_COLS + c;
      if (jj >= V) continue;
      out[(size_t)(t0 + g0 + r) * H * V + h * V + jj] = scan::tree_of_parts<PLAN>(o_s + r * parts * LT_COLS + c, parts, LT_COLS);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < LT_ROWS; ++i) {
    const int d = part * LT_ROWS + i;
    if (live && d < D) S[(size_t)d * V + j] = s[i];
  }
}

// ---- long portions -----------------------------------------------------------------------------------------------------
// The activated rows [q | k | v] of every token in 32-bit, once for all columns' blocks (16 bytes of input a thread).
template <typename T>
__global__ void __launch_bounds__(256)
lightning_activate_kernel(float* __restrict__ ready, const T* __restrict__ proj, int proj_stride, int width) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int PER16 = 16 / (int)sizeof(T);
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * PER16;
  if (c >= width) return;
  const uint4 raw = *reinterpret_cast<const uint4*>(proj + (size_t)blockIdx.x * proj_stride + c);
  const T* e = reinterpret_cast<const T*>(&raw);
  float* dst = ready + (size_t)blockIdx.x * width + c;
#pragma unroll
  for (int u = 0; u < PER16; u += 4)
    *reinterpret_cast<float4*>(dst + u) = make_float4(act_silu<T>(to_f(e[u])), act_silu<T>(to_f(e[u + 1])),
                                                      act_silu<T>(to_f(e[u + 2])), act_silu<T>(to_f(e[u + 3])));
}

// Half a warp owns a column, a lane ROWS rows of it, in registers over all tokens.  Groups of 16 tokens arrive by cp.async,
// two groups ahead, issued by two warps of their own (the copies of a group cost a computing warp a quarter of its time); a
// column's 16 outputs of a group are summed over the lanes at once.  What bounds it: a warp alone on its scheduler (portions of
// one request have 768 columns for 592 schedulers), about 35 instructions and 125 cycles a token.  2,048 tokens, 6 heads of
// 128 x 128, activation included: 350 -> 135 us (before: a thread a column and 8 rows, a block-wide sum of its parts, the
// activation in every block of 16 columns).
constexpr int LL_WARPS = 4, LL_LOAD_WARPS = 2, LL_COLS = 2 * LL_WARPS, LL_STAGES = 3;

template <int ROWS>
__global__ void __launch_bounds__((LL_WARPS + LL_LOAD_WARPS) * 32, 1)
lightning_long_kernel(float* __restrict__ out, const float* __restrict__ ready, float* __restrict__ state,
                      const float* __restrict__ decay, const int* __restrict__ q_start, const int* __restrict__ slots, int H,
                      int D, int V) {
  using namespace scan;
  constexpr int DP = 16 * ROWS, TOK = 2 * DP + LL_COLS;
  static_assert(LT_GROUP == 16, "a group's outputs of a column are half a warp's lanes");
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float smem[];            // [LL_STAGES][LT_GROUP][DP q | DP k | LL_COLS v]
  const int h = blockIdx.y, b = blockIdx.z;
  const int t0 = q_start[b], n = q_start[b + 1] - t0;
  if (n <= 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = lane & 15, col = 2 * warp + (lane >> 4);
  const int j0 = blockIdx.x * LL_COLS, j = j0 + col;
  const int W = H * (2 * D + V);
  if (D < DP || j0 + LL_COLS > V) {
    for (int i = threadIdx.x; i < LL_STAGES * LT_GROUP * TOK / 4; i += blockDim.x)
      reinterpret_cast<float4*>(smem)[i] = make_float4(0.f, 0.f, 0.f, 0.f);    // (rows beyond D, columns beyond V stay zero)
    __syncthreads();
  }
  if (warp >= LL_WARPS) {
    // Loading warp w brings tokens w, w + LL_LOAD_WARPS, ... of a group, a lane the pieces lane, lane + 32 of q and k; the
    // first lanes the values.
    const int w = warp - LL_WARPS;
    const int chunks = D / 4, v_chunks = min(LL_COLS, V - j0) / 4;
    const float* src = ready + (size_t)(t0 + w) * W + h * D + 4 * lane;
    const float* v_src = ready + (size_t)(t0 + w) * W + 2 * H * D + h * V + j0 + 4 * lane;
    auto fetch = [&](int g0, int st) {
      const int gn = n - g0;
      const size_t first = (size_t)g0 * W;
      float* dst = smem + (st * LT_GROUP + w) * TOK;
#pragma unroll
      for (int rr = 0; rr < LT_GROUP / LL_LOAD_WARPS; ++rr) {
        if (w + rr * LL_LOAD_WARPS >= gn) break;
        const size_t off = first + (size_t)rr * LL_LOAD_WARPS * W;
        float* d = dst + rr * LL_LOAD_WARPS * TOK;
#pragma unroll
        for (int c = 0; c < DP / 4; c += 32) {
          if (lane + c < chunks) {
            const int at = 4 * piece_at<ROWS>(lane + c);
            cp_async_16(d + at, src + off + 4 * c, true);
            cp_async_16(d + DP + at, src + off + 4 * c + H * D, true);
          }
        }
        if (lane < v_chunks) cp_async_16(d + 2 * DP + 4 * lane, v_src + off, true);
      }
    };
#pragma unroll
    for (int st = 0; st < LL_STAGES - 1; ++st) {
      if (st * LT_GROUP < n) fetch(st * LT_GROUP, st);
      cp_async_commit();
    }
    int st = 0;
    for (int g0 = 0; g0 < n; g0 += LT_GROUP, st = st + 1 == LL_STAGES ? 0 : st + 1) {
      cp_async_wait<LL_STAGES - 2>();
      __syncthreads();                                     // group g0 is here, and the one before has been computed from
      const int ahead = g0 + (LL_STAGES - 1) * LT_GROUP;
      if (ahead < n) fetch(ahead, st == 0 ? LL_STAGES - 1 : st - 1);
      cp_async_commit();
    }
    cp_async_wait<0>();
    return;
  }
  const bool live = j < V;
  const float lam = decay[h];
  const f2 lam2 = pack2(lam, lam);
  float* S = state + ((size_t)slots[b] * H + h) * D * V + j;
  f2 s[ROWS / 2];
#pragma unroll
  for (int i = 0; i < ROWS / 2; ++i) {
    const int d = p * ROWS + 2 * i;                        // (D is a multiple of 4: both rows or none)
    const bool there = live && d < D;
    s[i] = pack2(there ? S[(size_t)d * V] : 0.f, there ? S[(size_t)(d + 1) * V] : 0.f);
  }
  float x[16];                                             // this lane's share of the column's 16 outputs
  struct Token {
    f2 q[ROWS / 2], k[ROWS / 2];
    float v;
  };
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem);
  const int v_at = p * ROWS < D ? 2 * DP + col : 4 * 15;   // (a lane of absent rows: the last lane's query row, which is zero)
  const bool second = p * ROWS + 8 < D;
  auto load = [&](Token& t, uint32_t at) {
    load_rows<ROWS>(at, p, t.q);
    load_rows<ROWS>(at + 4 * DP, p, t.k);
    t.v = load_f32(at + 4 * v_at);
  };
  auto take = [&](const Token& t, int r, Token& next, uint32_t next_at, bool more) {
    const f2 v2 = pack2(t.v, t.v);
    f2 kv[ROWS / 2];
#pragma unroll
    for (int i = 0; i < ROWS / 2; ++i) kv[i] = mul2_first(t.k[i], v2);
    if (more) load(next, next_at);
#pragma unroll
    for (int i = 0; i < ROWS / 2; ++i) s[i] = fma2(lam2, s[i], kv[i]);
    x[r] = dot_rows<ROWS>(s, t.q, 0.f, second);
  };
  int st = 0;
  for (int g0 = 0; g0 < n; g0 += LT_GROUP, st = st + 1 == LL_STAGES ? 0 : st + 1) {
    __syncthreads();
    const uint32_t grp = ring + 4 * st * LT_GROUP * TOK;
    const int gn = min(LT_GROUP, n - g0);
    Token tk[2];
    if (gn == LT_GROUP) {
      load(tk[0], grp);
#pragma unroll
      for (int r = 0; r < LT_GROUP; ++r) take(tk[r & 1], r, tk[(r + 1) & 1], grp + 4 * (r + 1) * TOK, r + 1 < LT_GROUP);
    } else {
#pragma unroll
      for (int r = 0; r < LT_GROUP; ++r) {
        x[r] = 0.f;
        if (r < gn) {
          load(tk[0], grp + 4 * r * TOK);
          take(tk[0], r, tk[1], 0, false);
        }
      }
    }
    const float o = sum_scatter(x, lane);
    if (live && p < gn) out[(size_t)(t0 + g0 + p) * H * V + h * V + j] = o;
  }
#pragma unroll
  for (int i = 0; i < ROWS / 2; ++i) {
    const int d = p * ROWS + 2 * i;
    if (!live || d >= D) continue;
    const float2 v = unpack2(s[i]);
    S[(size_t)d * V] = v.x;
    S[(size_t)(d + 1) * V] = v.y;
  }
}

}  // namespace

// proj: [T, proj_stride] rows holding q at column 0, k at H D, v at 2 H D.  state: [slots, H, D, V] 32-bit.
// decay: [H] 32-bit on the device.  out: [T, H V] 32-bit.
// T: tokens of all requests.  longest: the most tokens a request brings (0: not known); from LT_LATE_TOKENS on the kernel is
// launched late (see ts_launch_late).
// ts_lightning_long takes portions from LL_TOKENS on where ts_lightning_long_supported says so, with ready [T, H (2 D + V)]
// 32-bit as work memory; outputs and states are the same bits.  (From how
// many tokens on its second launch pays is the caller's to say.)
constexpr int LT_LATE_TOKENS = 64, LL_TOKENS = 128;

TS_API int ts_lightning_ex(float* out, const void* proj, int proj_stride, float* state, const float* decay,
                           const int* q_start, const int* slots, int B, int T, int H, int D, int V, int longest, int dtype,
                           void* stream);

TS_API int ts_lightning(float* out, const void* proj, int proj_stride, float* state, const float* decay,
                        const int* q_start, const int* slots, int B, int H, int D, int V, int dtype, void* stream) {
  return ts_lightning_ex(out, proj, proj_stride, state, decay, q_start, slots, B, 0, H, D, V, 0, dtype, stream);
}

TS_API int ts_lightning_ex(float* out, const void* proj, int proj_stride, float* state, const float* decay,
                           const int* q_start, const int* slots, int B, int T, int H, int D, int V, int longest, int dtype,
                           void* stream) {
  if (B <= 0) return 0;
  if (H <= 0 || D <= 0 || V <= 0) TS_REFUSE(TS_ERR_SHAPE, "ts_lightning: %d heads of %d x %d", H, D, V);
  const int parts = ceil_div(D, LT_ROWS);
  if (parts * LT_COLS > 512) TS_REFUSE(TS_ERR_LIMIT, "ts_lightning: keys of %d (limit %d)", D, 512 / LT_COLS * LT_ROWS);
  if (B > 65535 || H > 65535) TS_REFUSE(TS_ERR_LIMIT, "ts_lightning: %d requests / %d heads per launch", B, H);
  cudaStream_t s = (cudaStream_t)stream;
  const int elem = dtype == TS_F32 ? 4 : 2, per16 = 16 / elem;
  // asynchronous 16-byte copies of the raw rows: every piece of a row (q, k, this block's v columns) must start on
  // a 16-byte boundary in global and in shared memory
  const int fast_rows = D % per16 == 0 && V % per16 == 0 && proj_stride % per16 == 0 && !((uintptr_t)proj & 15);
  const size_t smem = sizeof(float) * LT_GROUP * ((size_t)2 * parts * LT_ROWS + LT_COLS + (size_t)parts * LT_COLS) +
                      (size_t)2 * LT_GROUP * (2 * D + LT_COLS) * elem;
  dim3 grid(ceil_div(V, LT_COLS), H, B);
  // Portions of 64 tokens or more go to the planned instance while the chip holds all its blocks at once (512 threads an SM).  6
  // heads of 128 x 128, planned against lean: 127 tokens 24.1 / 26.9 us, 383 tokens of 6 requests 89 / 101, of 8 requests 147 /
  // 136, 256 tokens beside 8 single ones 55 / 52; of 64 x 64, 383 tokens 58 / 75.  Keys over 128 wide count requests by their length,
  // because one of their blocks fills an SM either way (383 tokens beside 8 single ones 98 / 106).
  const long long room = 512LL * ts_sm_count(), threads = (long long)grid.x * H * parts * LT_COLS;
  const bool planned = longest >= LT_LATE_TOKENS && (threads * B <= room || (parts > 16 && threads * T <= room * longest));
#define TS_LT(TT)                                                                                                   \
  do {                                                                                                              \
    static size_t configured = 0;                                                                                   \
    if (smem > 48 * 1024 && smem > configured) {                                                                    \
      cudaError_t e = cudaFuncSetAttribute(lightning_kernel<TT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e == cudaSuccess)                                                                                         \
        e = cudaFuncSetAttribute(lightning_kernel<TT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e != cudaSuccess) TS_REFUSE((int)e, "ts_lightning: shared memory %zu: %s", smem, cudaGetErrorString(e)); \
      configured = smem;                                                                                            \
    }                                                                                                               \
    if (planned)                                                                                                    \
      ts_launch_late(lightning_kernel<TT, true>, dim3(grid), dim3(parts * LT_COLS), smem, s, out, (const TT*)proj, proj_stride, \
                     state, decay, q_start, slots, H, D, V, parts, fast_rows);                                      \
    else if (longest >= LT_LATE_TOKENS)                                                                             \
      ts_launch_late(lightning_kernel<TT, false>, dim3(grid), dim3(parts * LT_COLS), smem, s, out, (const TT*)proj, proj_stride, \
                     state, decay, q_start, slots, H, D, V, parts, fast_rows);                                      \
    else                                                                                                            \
      ts_launch(lightning_kernel<TT, false>, dim3(grid), dim3(parts * LT_COLS), smem, s, out, (const TT*)proj, proj_stride, \
                state, decay, q_start, slots, H, D, V, parts, fast_rows);                                           \
  } while (0)
  if (dtype == TS_F32) TS_LT(float);
  else if (dtype == TS_BF16) TS_LT(bf16);
  else TS_REFUSE(TS_ERR_DTYPE, "ts_lightning: dtype %d", dtype);
#undef TS_LT
  TS_LAUNCH_CHECK();
}

TS_API int ts_lightning_long_supported(int D, int V, int proj_stride, int longest, int dtype) {
  const int per16 = dtype == TS_F32 ? 4 : 8;
  return (dtype == TS_F32 || dtype == TS_BF16) && longest >= LL_TOKENS && D > 0 && D <= 256 && D % per16 == 0 && V > 0 &&
         V % per16 == 0 && proj_stride % per16 == 0;
}

TS_API int ts_lightning_long(float* out, const void* proj, int proj_stride, float* ready, float* state, const float* decay,
                             const int* q_start, const int* slots, int B, int T, int H, int D, int V, int longest, int dtype,
                             void* stream) {
  if (B <= 0 || T <= 0) return 0;
  if (H <= 0 || !ts_lightning_long_supported(D, V, proj_stride, longest, dtype) || (((uintptr_t)proj | (uintptr_t)ready) & 15))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_lightning_long: %d heads of %d x %d, rows of %d", H, D, V, proj_stride);
  if (B > 65535 || H > 65535) TS_REFUSE(TS_ERR_LIMIT, "ts_lightning_long: %d requests / %d heads per launch", B, H);
  cudaStream_t s = (cudaStream_t)stream;
  const int width = H * (2 * D + V);
  const dim3 act(T, ceil_div(width, 256 * (dtype == TS_F32 ? 4 : 8)));
  if (act.y > 65535) TS_REFUSE(TS_ERR_LIMIT, "ts_lightning_long: rows of %d", width);
  const dim3 grid(ceil_div(V, LL_COLS), H, B);
#define TS_LL(RR)                                                                                                    \
  do {                                                                                                               \
    constexpr size_t smem = sizeof(float) * LL_STAGES * LT_GROUP * (2 * 16 * RR + LL_COLS);                          \
    static bool configured = false;                                                                                  \
    if (!configured) {                                                                                               \
      cudaError_t e = cudaFuncSetAttribute(lightning_long_kernel<RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e != cudaSuccess) TS_REFUSE((int)e, "ts_lightning_long: shared memory %zu: %s", smem, cudaGetErrorString(e)); \
      configured = true;                                                                                             \
    }                                                                                                                \
    ts_launch_late(lightning_long_kernel<RR>, grid, dim3((LL_WARPS + LL_LOAD_WARPS) * 32), smem, s, out, ready, state, decay, \
                   q_start, slots, H, D, V);                                                                         \
  } while (0)
  if (dtype == TS_F32) ts_launch(lightning_activate_kernel<float>, act, dim3(256), 0, s, ready, (const float*)proj, proj_stride, width);
  else ts_launch(lightning_activate_kernel<bf16>, act, dim3(256), 0, s, ready, (const bf16*)proj, proj_stride, width);
  if (D <= 128) TS_LL(8);
  else TS_LL(16);
#undef TS_LL
  TS_LAUNCH_CHECK();
}
