// Attention of requests that bring ONE token, over few enough (request, kv head) pairs that the launch's latency counts:
// plain grouped-query attention, the attention with options of attention_biased.cu (capped scores, distance bias, window,
// blocks, kept first tokens, sinks, gated and turned outputs) and latent rows that hold their values.  bfloat16.
//
// Counterpart of the reference's split-K flash-decoding kernels (turingserve/ops/triton_decode_attention.py:60-163).
//
// The keys of a pair are cut over the blocks of one thread-block cluster, as large a cluster as lets all pairs run at
// once.  What such a launch costs is a chain of latencies (with 2,048 keys a request all there is to read is 2.6 us at 8
// requests), so: the first keys and values, up to 320 a block, are in shared memory before the wait for the kernel before is
// over, all but the new token's row, where the caller vouches that nothing queued before the step still writes what is read then
// (`early`: the wait for one kernel is not a wait for those before it, as every kernel releases its successor at its start);
// no barrier stands between a warp and its keys (64 and 128 columns); and the blocks' sums
// cross the cluster once, pushed to the block that finishes a share of the output, as a read of a peer's shared memory costs a
// round trip of 0.5 us and more.  The weights enter the second product as one bfloat16 term (P2 false: plain attention, as in
// the reference) or as two.
//
// Measured (captured, keys from DRAM, us a launch; against the kernels that took these calls before): 12 heads over 2 of 128,
// 8 requests of 300 / 1,000 / 2,048 / 6,000 keys 4.0 / 5.8 / 7.6 / 13.3, before 6.6 / 8.6 / 10.5 / 18.4; 1 request of 2,048
// 5.0 / 8.6; 32 requests of 2,048 14.3 / 17.0; 14 heads over 2 of 64, 1 request of 1,000 3.2 / 5.7; with cap, bias and window
// of 1,024, 8 requests 6.4 / 14.9; latent rows: see below.  Not `early`: 0.2 to 1.5 us more (capped, 8 x 2,048 6.6 -> 7.6;
// latent 16.3 -> 17.6).
#include "common.cuh"
#include "mma_utils.cuh"

namespace {

constexpr float SG_LOG2E = 1.4426950408889634f;
constexpr int SG_MAX_CLUSTER = 16;

__device__ __forceinline__ float capped(float s, float cap, float inv_cap) {
  const float t = __expf(2.f * s * inv_cap);
  return cap * (1.f - __fdividef(2.f, t + 1.f));
}

struct SingleArgs {
  bf16* out;
  int out_ts, out_hs;
  const bf16* q;
  int q_ts, q_hs;
  const bf16* k_cache;
  const bf16* v_cache;
  const int* block_tables;
  const int* q_start;
  const int* seq_lens;
  int table_width, H, KVH, page;
  float scale, softcap;
  const float* slopes;
  int window, block_of, keep;
  const float* sinks;
  AttnFinish fin;
  int early;              // nothing before this step's kernels still writes its arrays or older rows: they are read before the wait
};

__device__ __forceinline__ void st_peer_v4(unsigned addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_peer_v2(unsigned addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}

// What a head's sum over all blocks, relative to its maximum M with weights adding up to L, is multiplied by: one over the sum
// of weights, the sink among them, times the head's gate.
__device__ __forceinline__ float finish_factor(const SingleArgs& a, float M, float L, int row_q, int head) {
  float inv = 0.f;
  if (!(L <= 0.f)) {                                                       // (a NaN goes through)
    const float sk = a.sinks != nullptr ? a.sinks[head] * SG_LOG2E : -INFINITY;
    const float top = fmaxf(M, sk), down = exp2f(M - top);
    inv = down / (L * down + exp2f(sk - top));
  }
  if (a.fin.gate != nullptr) inv *= 1.f / (1.f + expf(-to_f(((const bf16*)a.fin.gate)[(size_t)row_q * a.fin.gate_ts + head])));
  return inv;
}

// -- latent rows -----------------------------------------------------------------------------------------------------------
// 512 columns of sums are too many for one warp, so the block goes through stages of keys together: scores by groups of 16
// keys and parts of the columns (mma.sync m16n8k16, the heads in the 16 or 32 rows), softmax a warp a head with the running
// maximum and sum in shared memory, second product a warp some columns over all of a stage's keys.  mma.sync bounds it: 1,000
// products of 16 x 8 x 16 for every 80 keys an SM.  12 heads over one, 8 requests of 300 / 1,000 / 2,048 keys 10.7 / 12.2 / 16.2 us,
// before 22.4 / 29.7 / 34.5; 48 requests of 2,048 52 / 124; 28 heads, 8 of 2,048 29 / 41.
// The sizes of an instance: stages of STAGE keys, two of them; NKP warps share a group of 16 keys' columns; CW columns of
// the values a warp.
template <int DK, int DV, bool V_IN_K, int MT, int STAGE, int NKP, int WARPS, int CW>
struct Shape {
  static constexpr int ROWS = 16 * MT, NKG = STAGE / 16, KPP = DK / 16 / NKP;
  static constexpr int K_BYTES = STAGE * DK * 2, V_BYTES = V_IN_K ? 0 : STAGE * DV * 2;
  static constexpr int SC_LD = STAGE + 8, P_LD = STAGE + 8;                // (rows apart by an odd number of 16-byte pieces)
  static constexpr size_t at_v = 2 * (size_t)K_BYTES, at_sc = at_v + 2 * (size_t)V_BYTES;
  static constexpr size_t at_p = at_sc + sizeof(float) * NKP * ROWS * SC_LD;
  static constexpr size_t at_m = at_p + 2 * (size_t)ROWS * P_LD * 2;       // m, l, corr [ROWS]
  static constexpr size_t at_ml = at_m + sizeof(float) * ROWS * 4;         // from the peers
  static constexpr size_t bytes = at_ml + sizeof(float2) * ROWS * SG_MAX_CLUSTER;
  static_assert(STAGE % 16 == 0 && DK % (16 * NKP) == 0 && NKG * NKP <= WARPS && DV % CW == 0 && DV / CW <= WARPS && CW % 16 == 0, "");
  static_assert((size_t)ROWS * (DV + 8 * SG_MAX_CLUSTER) * 4 <= at_sc, "the peers' sums stand in the stages' place");
};

template <int DK, int DV, bool V_IN_K, int MT, int STAGE, int NKP, int WARPS, int CW, bool P2>
__global__ void __launch_bounds__(WARPS * 32, 1) attention_single_kernel(const SingleArgs a) {
  pdl_launch_dependents();
  if (!a.early) pdl_wait();
  using S = Shape<DK, DV, V_IN_K, MT, STAGE, NKP, WARPS, CW>;
  constexpr int THREADS = WARPS * 32, CHK = DK / 8, CHV = DV / 8, NTW = CW / 8, PVW = DV / CW;
  extern __shared__ __align__(128) unsigned char smem[];
  const int rank = blockIdx.x, n_blocks = gridDim.x, kvh = blockIdx.y, b = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = a.H / a.KVH;
  const int seq_len = a.seq_lens[b], row_q = a.q_start[b], pos = seq_len - 1;
  float* sc = reinterpret_cast<float*>(smem + S::at_sc);                   // [NKP][ROWS][SC_LD]
  bf16* p_hi = reinterpret_cast<bf16*>(smem + S::at_p);                    // [ROWS][P_LD], then the second terms
  bf16* p_lo = p_hi + S::ROWS * S::P_LD;
  float* m_s = reinterpret_cast<float*>(smem + S::at_m);
  float* l_s = m_s + S::ROWS;
  float* corr_s = l_s + S::ROWS;

  // The visible keys, in order: the kept first tokens that lie before the window, then the window's (or all).
  int lo = a.window > 0 ? max(0, seq_len - a.window) : 0;
  if (a.block_of > 0 && seq_len > 0) lo = max(lo, pos / a.block_of * a.block_of);
  const int kept = a.keep > 0 ? min(a.keep, lo) : 0;
  const int n_keys = seq_len > 0 ? kept + seq_len - lo : 0;
  const int per = ((n_keys + n_blocks - 1) / n_blocks + 15) / 16 * 16;
  const int v0 = min(n_keys, rank * per), v1 = min(n_keys, v0 + per);      // this block's
  const int n_stages = (v1 - v0 + STAGE - 1) / STAGE;
  auto key_at = [&](int v) { return v < kept ? v : lo + v - kept; };

  // A key row's 16-byte pieces by LPK lanes; the pages of all of a thread's keys are looked up before any copy.
  constexpr int LPK = CHK >= 32 ? 32 : (CHK >= 16 ? 16 : 8), KPI = WARPS * (32 / LPK), RB = (STAGE + KPI - 1) / KPI;
  const int page_shift = (a.page & (a.page - 1)) == 0 ? 31 - __clz(a.page) : -1;
  const int* table = a.block_tables + (size_t)b * a.table_width;
  auto row_of = [&](int j) {
    const int lp = page_shift >= 0 ? (j >> page_shift) : (j / a.page);
    return make_int2(table[lp], j - lp * a.page);
  };
  auto load_stage = [&](int i, bool skip_new) {
    unsigned char* ks = smem + (size_t)(i & 1) * S::K_BYTES;
    unsigned char* vs = smem + S::at_v + (size_t)(i & 1) * S::V_BYTES;
    int2 at[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const int v = v0 + i * STAGE + r * KPI + warp * (32 / LPK) + lane / LPK;
      at[r] = v < v1 ? row_of(key_at(v)) : make_int2(0, 0);
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const int key = r * KPI + warp * (32 / LPK) + lane / LPK, v = v0 + i * STAGE + key;
      if (key >= STAGE || (skip_new && v == n_keys - 1)) continue;         // (the new token's row: after the wait)
      const bool ok = v < v1;                                              // (rows past the end are zeroed)
      const size_t tok = ((size_t)at[r].x * a.KVH + kvh) * a.page + at[r].y;
      const bf16* krow = a.k_cache + tok * DK;
#pragma unroll
      for (int c = lane % LPK; c < CHK; c += LPK) cp_async_16(ks + swz<DK>(key, c), krow + c * 8, ok);
      if constexpr (!V_IN_K) {
        const bf16* vrow = a.v_cache + tok * DV;
#pragma unroll
        for (int c = lane % LPK; c < CHV; c += LPK) cp_async_16(vs + swz<DV>(key, c), vrow + c * 8, ok);
      }
    }
  };
  if (n_stages > 0) load_stage(0, true);
  cp_async_commit();
  if (n_stages > 1) load_stage(1, true);
  cp_async_commit();
  // (rows without a head weigh nothing in any stage)
  for (int i = threadIdx.x; i < 2 * S::ROWS * S::P_LD / 8; i += THREADS) reinterpret_cast<uint4*>(p_hi)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = threadIdx.x; i < S::ROWS; i += THREADS) {
    m_s[i] = -INFINITY;
    l_s[i] = 0.f;
    corr_s[i] = 0.f;
  }
  pdl_wait();
  const int new_stage = v1 == n_keys && v1 > v0 ? (v1 - 1 - v0) / STAGE : -1;
  if (new_stage >= 0 && new_stage < 2) {
    const int2 at = row_of(pos);
    const size_t tok = ((size_t)at.x * a.KVH + kvh) * a.page + at.y;
    const int key = v1 - 1 - v0 - new_stage * STAGE;
    for (int c = threadIdx.x; c < CHK; c += THREADS)
      cp_async_16(smem + (size_t)new_stage * S::K_BYTES + swz<DK>(key, c), a.k_cache + tok * DK + c * 8, true);
    if constexpr (!V_IN_K)
      for (int c = threadIdx.x; c < CHV; c += THREADS)
        cp_async_16(smem + S::at_v + (size_t)new_stage * S::V_BYTES + swz<DV>(key, c), a.v_cache + tok * DV + c * 8, true);
  }
  cp_async_commit();

  const int kg = warp % S::NKG, kp = warp / S::NKG;
  unsigned qf[MT][S::KPP][4];
  if (kp < NKP) {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int r0 = m * 16 + (lane >> 2), r1 = r0 + 8;
      const bf16* q0 = a.q + (size_t)row_q * a.q_ts + (size_t)(kvh * G + r0) * a.q_hs + kp * S::KPP * 16 + (lane & 3) * 2;
      const bf16* q1 = q0 + (size_t)8 * a.q_hs;
#pragma unroll
      for (int ks = 0; ks < S::KPP; ++ks) {
        qf[m][ks][0] = r0 < G ? *reinterpret_cast<const unsigned*>(q0 + ks * 16) : 0u;
        qf[m][ks][1] = r1 < G ? *reinterpret_cast<const unsigned*>(q1 + ks * 16) : 0u;
        qf[m][ks][2] = r0 < G ? *reinterpret_cast<const unsigned*>(q0 + ks * 16 + 8) : 0u;
        qf[m][ks][3] = r1 < G ? *reinterpret_cast<const unsigned*>(q1 + ks * 16 + 8) : 0u;
      }
    }
  }
  float o[MT][NTW][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int i = 0; i < NTW; ++i) o[m][i][0] = o[m][i][1] = o[m][i][2] = o[m][i][3] = 0.f;
  const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
  const int mat = lane >> 3, mr = lane & 7;

  for (int i = 0; i < n_stages; ++i) {
    // groups of copies, oldest first: the first two stages, the new row, then one per iteration
    if (i == 0 && new_stage != 0 && n_stages > 1) cp_async_wait<2>();
    else if (i == 0) cp_async_wait<0>();
    else cp_async_wait<1>();
    __syncthreads();
    const unsigned char* ks_ = smem + (size_t)(i & 1) * S::K_BYTES;
    const unsigned char* vs_ = V_IN_K ? ks_ : smem + S::at_v + (size_t)(i & 1) * S::V_BYTES;
    const int left = v1 - v0 - i * STAGE;                                  // keys from this stage on
    if (kp < NKP && kg * 16 < left) {
      float s[MT][2][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[m][0][e] = s[m][1][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < S::KPP; ++ks) {
        unsigned b0, b1, b2, b3;
        ldmatrix_x4(b0, b1, b2, b3, ks_ + swz<DK>(kg * 16 + (mat >> 1) * 8 + mr, (kp * S::KPP + ks) * 2 + (mat & 1)));
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          mma_bf16(s[m][0], qf[m][ks], b0, b1);
          mma_bf16(s[m][1], qf[m][ks], b2, b3);
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int n = 0; n < 2; ++n)
            *reinterpret_cast<float2*>(sc + (kp * S::ROWS + m * 16 + (lane >> 2) + 8 * h) * S::SC_LD + kg * 16 + n * 8 + (lane & 3) * 2) =
                make_float2(s[m][n][2 * h], s[m][n][2 * h + 1]);
    }
    __syncthreads();
    for (int row = warp; row < G; row += WARPS) {
      constexpr int NK = (STAGE + 31) / 32;
      const float slope = a.slopes != nullptr ? a.slopes[kvh * G + row] : 0.f;
      const float* mine = sc + row * S::SC_LD;
      float v[NK], mx = -INFINITY;
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        const int key = n * 32 + lane;
        v[n] = -INFINITY;
        if (key < STAGE && key < left) {
          float x = mine[key];
#pragma unroll
          for (int k = 1; k < NKP; ++k) x += mine[k * S::ROWS * S::SC_LD + key];
          x *= a.scale;
          if (a.softcap > 0.f) x = capped(x, a.softcap, inv_cap);
          v[n] = (x - slope * (float)(pos - key_at(v0 + i * STAGE + key))) * SG_LOG2E;
        }
        mx = fmaxf(mx, v[n]);
      }
      mx = warp_max(mx);
      const float m_old = m_s[row], m_new = fmaxf(m_old, mx);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < NK; ++n) {
        const int key = n * 32 + lane;
        const float p = exp2f(v[n] - m_use);
        sum += p;
        if (key < STAGE) {
          const bf16 hi = __float2bfloat16_rn(p);
          p_hi[row * S::P_LD + key] = hi;
          if constexpr (P2) p_lo[row * S::P_LD + key] = __float2bfloat16_rn(p - to_f(hi));
        }
      }
      sum = warp_sum(sum);
      __syncwarp();
      if (lane == 0) {
        const float corr = exp2f(m_old - m_use);
        corr_s[row] = corr;
        m_s[row] = m_new;
        l_s[row] = l_s[row] * corr + sum;
      }
    }
    __syncthreads();
    if (warp < PVW) {
      if (i > 0) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float c0 = corr_s[m * 16 + (lane >> 2)], c1 = corr_s[m * 16 + (lane >> 2) + 8];
#pragma unroll
          for (int n = 0; n < NTW; ++n) {
            o[m][n][0] *= c0;
            o[m][n][1] *= c0;
            o[m][n][2] *= c1;
            o[m][n][3] *= c1;
          }
        }
      }
      const int groups = min(S::NKG, (left + 15) >> 4);
#pragma unroll 2
      for (int kk = 0; kk < groups; ++kk) {
        unsigned hi[MT][4], lw[MT][4];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const int at = (m * 16 + (mat & 1) * 8 + mr) * S::P_LD + kk * 16 + (mat >> 1) * 8;
          ldmatrix_x4(hi[m][0], hi[m][1], hi[m][2], hi[m][3], p_hi + at);
          if constexpr (P2) ldmatrix_x4(lw[m][0], lw[m][1], lw[m][2], lw[m][3], p_lo + at);
        }
#pragma unroll
        for (int n = 0; n < NTW; n += 2) {
          unsigned b0, b1, b2, b3;
          ldmatrix_x4_trans(b0, b1, b2, b3, vs_ + swz<V_IN_K ? DK : DV>(kk * 16 + (mat & 1) * 8 + mr, warp * (CW / 8) + n + (mat >> 1)));
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            mma_bf16(o[m][n], hi[m], b0, b1);
            mma_bf16(o[m][n + 1], hi[m], b2, b3);
            if constexpr (P2) {
              mma_bf16(o[m][n], lw[m], b0, b1);
              mma_bf16(o[m][n + 1], lw[m], b2, b3);
            }
          }
        }
      }
    }
    __syncthreads();
    if (i + 2 < n_stages) load_stage(i + 2, false);
    cp_async_commit();
  }
  cp_async_wait<0>();
  // All blocks of the cluster are done with their stages: the sums go from registers to where they are finished, eight columns
  // nt to block nt % n, with the heads' (m, l) to all, into the stages' place.
  if (n_blocks > 1) cluster_sync_all();
  else __syncthreads();
  constexpr int NTS = DV / 8;
  const int room = (NTS + n_blocks - 1) / n_blocks;                        // groups of eight columns a block finishes
  float* in_o = reinterpret_cast<float*>(smem);                            // [blocks][ROWS][room][8]
  float2* in_ml = reinterpret_cast<float2*>(smem + S::at_ml);              // [blocks][ROWS]
  if (warp < PVW) {
#pragma unroll
    for (int n = 0; n < NTW; ++n) {
      const int nt = warp * NTW + n, to = nt % n_blocks, slot = nt / n_blocks;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = m * 16 + (lane >> 2) + 8 * h;
          if (row < G)
            st_peer_v2(peer_shared(in_o + ((size_t)(rank * S::ROWS + row) * room + slot) * 8 + (lane & 3) * 2, to),
                       make_float2(o[m][n][2 * h], o[m][n][2 * h + 1]));
        }
    }
  }
  for (int i = threadIdx.x; i < G * n_blocks; i += THREADS)
    st_peer_v2(peer_shared(in_ml + rank * S::ROWS + i % G, i / G), make_float2(m_s[i % G], l_s[i % G]));
  if (n_blocks > 1) cluster_sync_all();
  else __syncthreads();
  const int cols = (NTS - rank + n_blocks - 1) / n_blocks;                 // this block's groups: rank, rank + n, ...
  for (int idx = threadIdx.x; idx < G * cols * 2; idx += THREADS) {
    const int part = idx & 1, slot = (idx >> 1) % cols, row = (idx >> 1) / cols;
    float M = -INFINITY, L = 0.f;
    for (int s = 0; s < n_blocks; ++s) M = fmaxf(M, in_ml[s * S::ROWS + row].x);
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int s = 0; s < n_blocks; ++s) {
      const float2 ml = in_ml[s * S::ROWS + row];
      const float f = ml.x == -INFINITY ? 0.f : exp2f(ml.x - M);
      const float4 v = *reinterpret_cast<const float4*>(in_o + ((size_t)(s * S::ROWS + row) * room + slot) * 8 + part * 4);
      L = fmaf(ml.y, f, L);
      x.x = fmaf(v.x, f, x.x);
      x.y = fmaf(v.y, f, x.y);
      x.z = fmaf(v.z, f, x.z);
      x.w = fmaf(v.w, f, x.w);
    }
    const float inv = finish_factor(a, M, L, row_q, kvh * G + row);
    bf16* dst = a.out + (size_t)row_q * a.out_ts + (size_t)(kvh * G + row) * a.out_hs + (rank + slot * n_blocks) * 8 + part * 4;
    *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(x.x * inv, x.y * inv);
    *reinterpret_cast<__nv_bfloat162*>(dst + 2) = __floats2bfloat162_rn(x.z * inv, x.w * inv);
  }
}

// -- keys and values of 64 or 128 columns --------------------------------------------------------------------------------
// A warp takes whole tiles of 16 keys, the tiles of a block in turn, through two places of its own in shared memory: no
// barrier until its keys are done.  The heads are the products' narrow side (HT times 8 of them): S^T = K Q^T, and
// O^T += V^T P^T with the weights turned in registers, so that six or seven heads cost one product of 8 and 32 accumulators.
constexpr int SG_WARPS = 10, SG_SLOTS = 2;

template <int D, int HT>
struct Tiles {
  static constexpr int TILE_BYTES = 2 * 16 * D * 2;                        // keys, then values
  static constexpr int O_LD = D + 4;
  static constexpr size_t ring = (size_t)SG_WARPS * SG_SLOTS * TILE_BYTES;
  static constexpr size_t sums = sizeof(float) * SG_WARPS * HT * 8 * O_LD;  // the warps' sums, in the ring's place
  static constexpr size_t at_ml = ring > sums ? ring : sums;               // [WARPS][16] (m, l)
  static constexpr size_t at_in = at_ml + sizeof(float2) * SG_WARPS * 16;  // from the peers: [16 blocks][16 heads] (m, l), then pieces
  static constexpr size_t at_pieces = at_in + sizeof(float2) * SG_MAX_CLUSTER * 16;
  static constexpr size_t bytes = at_pieces + sizeof(float) * HT * 8 * D + 16 * SG_MAX_CLUSTER * 2;
};

__device__ __forceinline__ unsigned turned(unsigned x) {
  unsigned y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
template <int D, int HT, bool P2>
__global__ void __launch_bounds__(SG_WARPS * 32, HT == 1 ? 2 : 1) attention_single_tiles_kernel(const SingleArgs a) {
  pdl_launch_dependents();
  if (gridDim.x > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (this block runs: its shared memory may be written)
  if (!a.early) pdl_wait();
  using S = Tiles<D, HT>;
  constexpr int THREADS = SG_WARPS * 32, CH = D / 8, KS = D / 16, MD = D / 16;
  extern __shared__ __align__(128) unsigned char smem[];
  const int rank = blockIdx.x, n_blocks = gridDim.x, kvh = blockIdx.y, b = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, mat = lane >> 3, mr = lane & 7;
  const int G = a.H / a.KVH;
  const int seq_len = a.seq_lens[b], row_q = a.q_start[b], pos = seq_len - 1;

  // The visible keys, in order: the kept first tokens that lie before the window, then the window's (or all).
  int lo = a.window > 0 ? max(0, seq_len - a.window) : 0;
  if (a.block_of > 0 && seq_len > 0) lo = max(lo, pos / a.block_of * a.block_of);
  const int kept = a.keep > 0 ? min(a.keep, lo) : 0;
  const int n_keys = seq_len > 0 ? kept + seq_len - lo : 0;
  const int all_tiles = (n_keys + 15) >> 4, base = all_tiles / n_blocks, rem = all_tiles % n_blocks;
  const int first = rank * base + min(rank, rem), n_tiles = base + (rank < rem ? 1 : 0);       // this block's tiles of 16
  const int mine = n_tiles > warp ? (n_tiles - warp - 1) / SG_WARPS + 1 : 0;                   // this warp's: warp, warp + WARPS, ...
  auto key_at = [&](int v) { return v < kept ? v : lo + v - kept; };
  const int page_shift = (a.page & (a.page - 1)) == 0 ? 31 - __clz(a.page) : -1;
  const int* table = a.block_tables + (size_t)b * a.table_width;
  unsigned char* own = smem + (size_t)warp * SG_SLOTS * S::TILE_BYTES;
  // where key v of the request lies, in rows of the cache
  auto row_of = [&](int v) {
    const int j = key_at(v);
    const int lp = page_shift >= 0 ? (j >> page_shift) : (j / a.page);
    return ((size_t)table[lp] * a.KVH + kvh) * a.page + (j - lp * a.page);
  };
  // tile i of this warp; the new token's row is left out when `skip_new`, rows past the end are zeroed
  auto load_tile = [&](int i, bool skip_new) {
    const int v0 = (first + warp + i * SG_WARPS) * 16;
    unsigned char* ks = own + (i & 1) * S::TILE_BYTES;
    const size_t at = lane < 16 && v0 + lane < n_keys ? row_of(v0 + lane) : 0;        // (one look-up a key)
    constexpr int PER = 32 / CH;                                                      // keys a pass
#pragma unroll
    for (int r = 0; r < 16 / PER; ++r) {
      const int key = r * PER + lane / CH, c = lane % CH;
      const size_t tok = __shfl_sync(0xffffffffu, at, key);
      const bool ok = v0 + key < n_keys;
      if (skip_new && v0 + key == n_keys - 1) continue;
      cp_async_16(ks + swz<D>(key, c), a.k_cache + tok * D + c * 8, ok);
      cp_async_16(ks + 16 * D * 2 + swz<D>(key, c), a.v_cache + tok * D + c * 8, ok);
    }
  };
#pragma unroll
  for (int i = 0; i < SG_SLOTS; ++i) {
    if (i < mine) load_tile(i, true);
    cp_async_commit();
  }
  pdl_wait();
  // the new token's row, where one of those tiles holds it
  const int new_tile = (n_keys - 1) >> 4, new_i = (new_tile - first - warp) / SG_WARPS;
  if (n_keys > 0 && new_tile >= first && new_tile < first + n_tiles && (new_tile - first) % SG_WARPS == warp && new_i < SG_SLOTS) {
    const int key = (n_keys - 1) & 15;
    const size_t tok = row_of(n_keys - 1);
    unsigned char* ks = own + new_i * S::TILE_BYTES;
    if (lane < CH) cp_async_16(ks + swz<D>(key, lane), a.k_cache + tok * D + lane * 8, true);
    if (lane < CH) cp_async_16(ks + 16 * D * 2 + swz<D>(key, lane), a.v_cache + tok * D + lane * 8, true);
  }
  cp_async_commit();

  unsigned qf[HT][KS][2];
#pragma unroll
  for (int h = 0; h < HT; ++h) {
    const bf16* q = a.q + (size_t)row_q * a.q_ts + (size_t)(kvh * G + h * 8 + g) * a.q_hs + 2 * t;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      qf[h][ks][0] = h * 8 + g < G ? *reinterpret_cast<const unsigned*>(q + ks * 16) : 0u;
      qf[h][ks][1] = h * 8 + g < G ? *reinterpret_cast<const unsigned*>(q + ks * 16 + 8) : 0u;
    }
  }
  float o[HT][MD][4];                                                      // dims 16 i + g, + 8 of heads 8 h + 2t, + 1
  float m_run[HT][2], l_run[HT][2], slope[HT][2];
#pragma unroll
  for (int h = 0; h < HT; ++h) {
#pragma unroll
    for (int i = 0; i < MD; ++i) o[h][i][0] = o[h][i][1] = o[h][i][2] = o[h][i][3] = 0.f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      m_run[h][e] = -INFINITY;
      l_run[h][e] = 0.f;
      slope[h][e] = a.slopes != nullptr && h * 8 + 2 * t + e < G ? a.slopes[kvh * G + h * 8 + 2 * t + e] : 0.f;
    }
  }
  const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;

  for (int i = 0; i < mine; ++i) {
    // groups of copies, oldest first: the first two tiles, the new row, then one per iteration
    if (i == 0 && new_i != 0 && mine > 1) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (i == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
    else asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const unsigned char* ks_ = own + (i & 1) * S::TILE_BYTES;
    const unsigned char* vs_ = ks_ + 16 * D * 2;
    const int v0 = (first + warp + i * SG_WARPS) * 16;
    float s[HT][2][4];                                                     // (two sums: half the chain)
#pragma unroll
    for (int h = 0; h < HT; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[h][0][e] = s[h][1][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      unsigned k[4];
      ldmatrix_x4(k[0], k[1], k[2], k[3], ks_ + swz<D>((mat & 1) * 8 + mr, ks * 2 + (mat >> 1)));
#pragma unroll
      for (int h = 0; h < HT; ++h) mma_bf16(s[h][ks & 1], k, qf[h][ks][0], qf[h][ks][1]);
    }
    unsigned hi[HT][2], lw[HT][2];
#pragma unroll
    for (int h = 0; h < HT; ++h) {
      float x[4], corr[2];
#pragma unroll
      for (int e = 0; e < 4; ++e) {                                        // key v0 + g (+ 8), head 2t + (e & 1)
        const int v = v0 + g + 8 * (e >> 1);
        float y = (s[h][0][e] + s[h][1][e]) * a.scale;
        if (a.softcap > 0.f) y = capped(y, a.softcap, inv_cap);
        x[e] = v < n_keys ? (y - slope[h][e & 1] * (float)(pos - key_at(v))) * SG_LOG2E : -INFINITY;
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float mx = fmaxf(x[e], x[e + 2]);
#pragma unroll
        for (int w = 4; w < 32; w <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
        const float m_new = fmaxf(m_run[h][e], mx);
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        corr[e] = exp2f(m_run[h][e] - m_use);
        m_run[h][e] = m_new;
        x[e] = exp2f(x[e] - m_use);
        x[e + 2] = exp2f(x[e + 2] - m_use);
        l_run[h][e] = l_run[h][e] * corr[e] + (x[e] + x[e + 2]);           // (this lane's keys; summed over the lanes at the end)
      }
      const __nv_bfloat162 a0 = __floats2bfloat162_rn(x[0], x[1]), a1 = __floats2bfloat162_rn(x[2], x[3]);
      hi[h][0] = turned(*reinterpret_cast<const unsigned*>(&a0));
      hi[h][1] = turned(*reinterpret_cast<const unsigned*>(&a1));
      if constexpr (P2) {
        lw[h][0] = turned(pack_bf16(x[0] - __low2float(a0), x[1] - __high2float(a0)));
        lw[h][1] = turned(pack_bf16(x[2] - __low2float(a1), x[3] - __high2float(a1)));
      }
      if (i > 0)
#pragma unroll
        for (int n = 0; n < MD; ++n) {
          o[h][n][0] *= corr[0];
          o[h][n][1] *= corr[1];
          o[h][n][2] *= corr[0];
          o[h][n][3] *= corr[1];
        }
    }
#pragma unroll
    for (int n = 0; n < MD; ++n) {
      unsigned v[4];
      ldmatrix_x4_trans(v[0], v[1], v[2], v[3], vs_ + swz<D>((mat >> 1) * 8 + mr, n * 2 + (mat & 1)));
#pragma unroll
      for (int h = 0; h < HT; ++h) {
        mma_bf16(o[h][n], v, hi[h][0], hi[h][1]);
        if constexpr (P2) mma_bf16(o[h][n], v, lw[h][0], lw[h][1]);
      }
    }
    __syncwarp();
    if (i + SG_SLOTS < mine) load_tile(i + SG_SLOTS, false);
    cp_async_commit();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* o_s = reinterpret_cast<float*>(smem);                             // [WARPS][heads][O_LD], in the ring's place
  float2* ml_s = reinterpret_cast<float2*>(smem + S::at_ml);
  float2* in_ml = reinterpret_cast<float2*>(smem + S::at_in);
  float4* in_o = reinterpret_cast<float4*>(smem + S::at_pieces);
#pragma unroll
  for (int h = 0; h < HT; ++h)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float l = l_run[h][e];
#pragma unroll
      for (int w = 4; w < 32; w <<= 1) l += __shfl_xor_sync(0xffffffffu, l, w);
      const int head = h * 8 + 2 * t + e;
      if (g == 0) ml_s[warp * 16 + head] = make_float2(m_run[h][e], l);
      float* to = o_s + (size_t)(warp * HT * 8 + head) * S::O_LD + g;
#pragma unroll
      for (int n = 0; n < MD; ++n) {
        to[n * 16] = o[h][n][e];
        to[n * 16 + 8] = o[h][n][e + 2];
      }
    }
  __syncthreads();
  // The block's sums go where they are finished: piece p (a head's four columns and, so that pairs can be turned, the four half
  // a row further) to block p % n of the cluster, the heads' (m, l) to all.
  constexpr int QD = D / 8, HALF = D / 2;
  const int pieces = G * QD, room = (pieces + n_blocks - 1) / n_blocks;    // of a block's share from each peer
  if (n_blocks > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int p = threadIdx.x; p < pieces; p += THREADS) {
    const int head = p / QD, d = (p % QD) * 4;
    float M = -INFINITY, L = 0.f;
#pragma unroll
    for (int w = 0; w < SG_WARPS; ++w) M = fmaxf(M, ml_s[w * 16 + head].x);
    float4 x[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
    for (int w = 0; w < SG_WARPS; ++w) {
      const float2 ml = ml_s[w * 16 + head];
      const float f = ml.x == -INFINITY ? 0.f : exp2f(ml.x - M);
      L = fmaf(ml.y, f, L);
      const float* from = o_s + (size_t)(w * HT * 8 + head) * S::O_LD + d;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(from + h * HALF);
        x[h].x = fmaf(v.x, f, x[h].x);
        x[h].y = fmaf(v.y, f, x[h].y);
        x[h].z = fmaf(v.z, f, x[h].z);
        x[h].w = fmaf(v.w, f, x[h].w);
      }
    }
    const unsigned to = peer_shared(in_o + 2 * ((size_t)rank * room + p / n_blocks), p % n_blocks);
    st_peer_v4(to, x[0]);
    st_peer_v4(to + 16, x[1]);
    for (int to_rank = p % QD; to_rank < n_blocks; to_rank += QD) st_peer_v2(peer_shared(in_ml + rank * 16 + head, to_rank), make_float2(M, L));
  }
  if (n_blocks > 1) cluster_sync_all();
  else __syncthreads();
  for (int k = threadIdx.x; k * n_blocks + rank < pieces; k += THREADS) {
    const int p = k * n_blocks + rank, head = p / QD, d = (p % QD) * 4;
    float M = -INFINITY, L = 0.f;
    for (int s = 0; s < n_blocks; ++s) M = fmaxf(M, in_ml[s * 16 + head].x);
    float4 x[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll 4
    for (int s = 0; s < n_blocks; ++s) {
      const float2 ml = in_ml[s * 16 + head];
      const float f = ml.x == -INFINITY ? 0.f : exp2f(ml.x - M);
      L = fmaf(ml.y, f, L);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = in_o[2 * ((size_t)s * room + k) + h];
        x[h].x = fmaf(v.x, f, x[h].x);
        x[h].y = fmaf(v.y, f, x[h].y);
        x[h].z = fmaf(v.z, f, x[h].z);
        x[h].w = fmaf(v.w, f, x[h].w);
      }
    }
    const float inv = finish_factor(a, M, L, row_q, kvh * G + head);
    float u[4] = {x[0].x * inv, x[0].y * inv, x[0].z * inv, x[0].w * inv}, w[4] = {x[1].x * inv, x[1].y * inv, x[1].z * inv, x[1].w * inv};
    if (a.fin.out_freq != nullptr) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float sn, cs;
        sincosf((float)pos * a.fin.out_freq[d + e], &sn, &cs);
        const float c = u[e], f = w[e];
        u[e] = c * cs + f * sn;
        w[e] = f * cs - c * sn;
      }
    }
    bf16* dst = a.out + (size_t)row_q * a.out_ts + (size_t)(kvh * G + head) * a.out_hs + d;
    *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(u[0], u[1]);
    *reinterpret_cast<__nv_bfloat162*>(dst + 2) = __floats2bfloat162_rn(u[2], u[3]);
    *reinterpret_cast<__nv_bfloat162*>(dst + HALF) = __floats2bfloat162_rn(w[0], w[1]);
    *reinterpret_cast<__nv_bfloat162*>(dst + HALF + 2) = __floats2bfloat162_rn(w[2], w[3]);
  }
}

// The largest cluster, up to `most`, of which the device holds `pairs` at once; more blocks than keys for them (128 each) are not asked for.
template <typename K>
int cluster_of(K kernel, int threads, size_t smem, int (&fits)[SG_MAX_CLUSTER + 1], int pairs, int reach, int most) {
  if (fits[1] < 0) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    for (int c = SG_MAX_CLUSTER; c >= 1; --c) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(c, 1, 1);
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)c;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int n = 0;
      const bool ok = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess;
      cudaGetLastError();                                                  // a refusal is an answer, not an error
      fits[c] = ok ? n : 0;
    }
  }
  int c = most;
  while (c > 1 && (pairs > fits[c] || (c - 1) * 128 >= reach)) --c;
  return c;
}

template <int D, int HT, bool P2>
int launch_tiles(const SingleArgs& a, int B, int reach, cudaStream_t s) {
  static int fits[SG_MAX_CLUSTER + 1] = {0, -1};
  const int c = cluster_of(attention_single_tiles_kernel<D, HT, P2>, SG_WARPS * 32, Tiles<D, HT>::bytes, fits, B * a.KVH, reach,
                           reach > 8 * SG_WARPS * SG_SLOTS * 16 ? SG_MAX_CLUSTER : 8);
  if (c == 0) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_single: %zu bytes of shared memory", Tiles<D, HT>::bytes);
  ts_launch_cluster(attention_single_tiles_kernel<D, HT, P2>, dim3(c, 1, 1), dim3(c, a.KVH, B), dim3(SG_WARPS * 32), Tiles<D, HT>::bytes, s, a);
  TS_LAUNCH_CHECK();
}

template <int DK, int DV, bool V_IN_K, int MT, int STAGE, int NKP, int WARPS, int CW, bool P2>
int launch(const SingleArgs& a, int B, int reach, cudaStream_t s) {
  using S = Shape<DK, DV, V_IN_K, MT, STAGE, NKP, WARPS, CW>;
  auto kernel = attention_single_kernel<DK, DV, V_IN_K, MT, STAGE, NKP, WARPS, CW, P2>;
  static int fits[SG_MAX_CLUSTER + 1] = {0, -1};
  const int c = cluster_of(kernel, WARPS * 32, S::bytes, fits, B * a.KVH, reach, reach > 8 * 2 * STAGE ? SG_MAX_CLUSTER : 8);
  if (c == 0) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_single: %zu bytes of shared memory", S::bytes);
  ts_launch_cluster(kernel, dim3(c, 1, 1), dim3(c, a.KVH, B), dim3(WARPS * 32), S::bytes, s, a);
  TS_LAUNCH_CHECK();
}

}  // namespace

// Whether the kernel has the widths: G heads a kv head, at most 16 (32 for latent rows).
TS_API int ts_attention_single_supported(int H, int KVH, int Dk, int Dv, int v_in_k, int dtype) {
  if (dtype != TS_BF16 || KVH <= 0 || H % KVH != 0) return 0;
  const int G = H / KVH;
  if (v_in_k) return Dk == 576 && Dv == 512 && G <= 32;
  return Dk == Dv && (Dk == 64 || Dk == 128) && G <= 16;
}

// Arguments as ts_attention_biased_mma's for requests of one token each.  reach: the most keys any of them sees.  two_terms:
// the weights enter the second product as two bfloat16 terms.  early: block_tables, q_start, seq_lens and the cache rows before
// each request's last were written by work that the stream has finished before the step's first kernel starts (a copy from the
// host stands between, say), so they are read before the wait for the kernel before; 0: after it.  TS_ERR_UNSUPPORTED: shapes, or strides off their boundaries, or
// clusters switched off.
TS_API int ts_attention_single(void* out, int out_ts, int out_hs, const void* q, int q_ts, int q_hs, const void* k_cache,
                               const void* v_cache, const int* block_tables, const int* q_start, const int* seq_lens, int B,
                               int table_width, int reach, int H, int KVH, int Dk, int Dv, int page, float scale, float softcap,
                               const float* slopes, int window, int block_of, const float* sinks, int keep, const float* out_freq,
                               const void* gate, int gate_ts, int two_terms, int early, void* stream) {
  if (B <= 0) return 0;
  const int v_in_k = v_cache == nullptr;
  if (!ts_attention_single_supported(H, KVH, Dk, Dv, v_in_k, TS_BF16) || !ts_clusters_enabled())
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_single: H=%d KVH=%d keys %d values %d", H, KVH, Dk, Dv);
  if ((q_ts % 2) || (q_hs % 2) || ((uintptr_t)q & 3) || (out_ts % 2) || (out_hs % 2) || ((uintptr_t)out & 3) ||
      (((uintptr_t)k_cache | (uintptr_t)v_cache) & 15))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_single: rows off their boundaries");
  if (B > 65535 || KVH > 65535) TS_REFUSE(TS_ERR_LIMIT, "ts_attention_single: %d requests / %d kv heads", B, KVH);
  if (keep < 0 || (keep > 0 && block_of > 0)) TS_REFUSE(TS_ERR_SHAPE, "ts_attention_single: %d kept tokens (with blocks of %d)", keep, block_of);
  SingleArgs a;
  a.out = (bf16*)out; a.out_ts = out_ts; a.out_hs = out_hs;
  a.q = (const bf16*)q; a.q_ts = q_ts; a.q_hs = q_hs;
  a.k_cache = (const bf16*)k_cache; a.v_cache = (const bf16*)v_cache;
  a.block_tables = block_tables; a.q_start = q_start; a.seq_lens = seq_lens;
  a.table_width = table_width; a.H = H; a.KVH = KVH; a.page = page;
  a.scale = scale; a.softcap = softcap; a.slopes = slopes;
  a.window = window; a.block_of = block_of; a.keep = keep; a.sinks = sinks;
  a.fin.out_freq = out_freq; a.fin.gate = gate; a.fin.gate_ts = gate_ts;
  a.early = early;
  cudaStream_t s = (cudaStream_t)stream;
  if (v_in_k && out_freq != nullptr) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_single: the pairs of latent values are not turned");
  if (v_in_k && H / KVH <= 16) return launch<576, 512, true, 1, 80, 3, 16, 32, true>(a, B, reach, s);
  if (v_in_k) return launch<576, 512, true, 2, 64, 4, 16, 32, true>(a, B, reach, s);
  const bool wide = H / KVH > 8;
#define TS_TILES(D, P2) return wide ? launch_tiles<D, 2, P2>(a, B, reach, s) : launch_tiles<D, 1, P2>(a, B, reach, s)
  if (Dk == 128 && two_terms) TS_TILES(128, true);
  if (Dk == 128) TS_TILES(128, false);
  if (two_terms) TS_TILES(64, true);
  TS_TILES(64, false);
#undef TS_TILES
}
