// The attention of attention_biased.cu (capped scores, distance bias per head, window, blocks of positions, a sink in the
// softmax's denominator, kept first tokens, outputs turned back and gated, values of their own or inside the key rows) for
// PROMPT PORTIONS on the 5th-generation tensor cores; bfloat16 storage, pages of a multiple of 16 tokens.
//
// One block = 128 query ROWS (a row is one (token, head-in-group) pair of one kv head) x DV value columns, keys TK (64 or
// 128) at a time.  Warps 0-7 are the softmax (a row = a tensor-memory lane belongs to two threads, half of every tile's keys
// each), warp 8 issues the products, warps 9 and 10 the TMA loads, as in attention_prefill_tc.cu.  What differs:
//   * scores are scaled, capped and biased in 32-bit, and the softmax weights enter the second product as TWO bfloat16
//     terms (p = hi + lo, two products), so they carry 16 bits of mantissa.  A thread writes both over its own scores;
//   * the two threads of a row exchange their maxima in 32-bit (scores of any size), over a barrier of their two warps;
//   * values inside the key rows (latent rows of 576 = 512 + 64): a key tile (72 KB) is both the first product's operand
//     and, its columns chunk * DV .., the second's.  Two such tiles and the 128 query rows (144 KB) do not fit a block's
//     shared memory together, so the first QT * 64 query columns live in TENSOR memory (beside O's 256 and S's 2 x 64
//     columns) and the first product reads its A operand from there for these k-steps.  Value rows wider than DV are cut
//     over blocks, which each redo the scores.  A tile's 64-column blocks that are no values of this block are free once
//     its scores are there, the value blocks only when its O product is done: two rings, and the scores begin with the
//     former;
//   * keys a block must not see are masked, and their value rows are cleared in shared memory before the second product
//     reads them: a weight of zero times whatever a page holds behind a request's last token must stay zero;
//   * the same holds for a key that some rows of the block see and others do not: in the tiles where that happens (those of
//     the block's own tokens and of the window's lower edge) infinities and NaN among the values are taken out before the
//     product and added at the end to the rows that see them, read from memory once more.  With the look at such
//     tiles' values calls of 95 and 220 us take 1.4 us and 3 us longer.
// Order of the products: S(0) S(1) O(0) S(2) O(1) S(3) ...: a tile's softmax runs beside the O of the tile before and the
// S of the tile behind.
//
// What bounds it (clock stamps in the kernel): a tile's chain.  576: 36 + 8 products of 46 to 128 cycles a tile of 64 keys (64
// rows of K give a product no fewer cycles than 128 would), 3,600 cycles from issue to completion of about 4,450 a tile (148
// blocks, 592 tokens of 16 heads behind 2,048 and 6,144: 2.27 us a tile more; by its counter the tensor pipe is active for 2,300
// of them), and some 20 us a launch for the blocks' start, masked tiles and end; 128: 2,900 cycles a tile of
// 128 keys, of which the softmax is busy for 2,400.  Portion of 2,048 tokens, 12 heads (L2 flushed), against the mma.sync
// kernel of attention_biased_mma.cu: latent rows 660 -> 164 us; 128 over 2 kv heads 149 -> 43 us, with cap and bias 174 ->
// 59 us; 64 over 2: 115 -> 39 us.  512 tokens behind 3,000, 28 heads: latent 1,456 -> 266 us, 128 over 4: 254 -> 61 us.
#include <type_traits>

#include "common.cuh"
#include "tc_utils.cuh"

namespace {

using namespace tc;

constexpr int TQ = 128;                                    // query rows per block = TMEM lanes
constexpr int UNIT = 64;                                   // keys per unit of loading: a tile is one or two of them
constexpr int BOX_ROWS = 16;                               // keys per TMA box at least
constexpr uint32_t BLK_Q = TQ * 128;                       // bytes of 64 columns of the query rows
constexpr float RESCALE_STEP = 8.f;                        // log2 of how far a maximum may run ahead of its reference
constexpr float LOG2E_F = 1.4426950408889634f;
constexpr int SOFTMAX_THREADS = 2 * TQ;
constexpr int THREADS = SOFTMAX_THREADS + 96;
constexpr int MMA_WARP = SOFTMAX_THREADS / 32, LOAD_WARP = MMA_WARP + 1;    // (two loading warps)

template <int DK, int DV, int TK, bool V_IN_K, int QT, bool MAPS = false>
struct Plan {
  static constexpr int KT = TK / 2, UNITS = TK / UNIT;     // keys of a tile per softmax thread; units of loading
  static constexpr uint32_t BLK_KV = TK * 128;             // bytes of 64 columns of a key / value tile
  static constexpr int KB = DK / 64, VB = DV / 64;         // 64-column blocks of a key row, of a block's value columns
  static constexpr int STAGES = 2;
  static constexpr uint32_t K_BYTES = KB * BLK_KV, V_BYTES = V_IN_K ? 0 : VB * BLK_KV;
  static constexpr uint32_t Q_BYTES = (KB - QT) * BLK_Q;
  static constexpr uint32_t S_COL = 0, O_COL = 2 * TK, Q_COL = O_COL + DV;
  static constexpr uint32_t COLS = Q_COL + QT * 32;
  static constexpr uint32_t TMEM_COLS = 512;               // (every instance needs more than 256: a block an SM)
  static constexpr int BARRIERS = 4 * STAGES + 2 + 2 + 3;
  static constexpr size_t SMEM = Q_BYTES + STAGES * (K_BYTES + V_BYTES) + (BARRIERS + 1) / 2 * 16 + 16 + 4 * TQ * sizeof(float);
  static_assert(COLS > 256 && COLS <= 512 && SMEM <= 227 * 1024, "a block's tensor or shared memory");
};

struct Args {
  bf16* out;
  float* out32;            // two score maps a head: rows [T, H, 2, DV] in place of `out`
  const bf16* q;
  const bf16* values;      // the rows the values lie in ([page, kv head, token], value_row wide), and for a block's slow path only
  int value_row;
  const int* block_tables;
  const int* q_start;
  const int* seq_lens;
  const float* slopes;
  const float* sinks;
  int out_ts, out_hs, q_ts, q_hs;
  int table_width, H, KVH, page, box;
  int run;                 // pages per tile when a tile is several pages (then the run maps are valid), else 0
  float scale, softcap;
  int window, block_of, keep, v_chunks;
  int min_rows;            // requests of so many rows or fewer are another kernel's
  AttnFinish fin;
  int* status;
};

template <int N> using Int = std::integral_constant<int, N>;

// Whether one of two bfloat16 values is an infinity or NaN (its exponent all ones: adding the exponent's last bit carries
// into the sign's place), and the pair with such values replaced by zero.
__device__ __forceinline__ uint32_t odd(uint32_t pair) { return ((pair & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }
__device__ __forceinline__ uint32_t without_odd(uint32_t pair) {
  const uint32_t o = odd(pair);
  return pair & ~(((o >> 15) & 0x00010001u) * 0xffffu);
}

// Adds to one row's stored result, columns [c0, c0 + n) and [c0 + half, c0 + half + n), the infinities and NaN among the values of
// the keys j it sees: from first on, lo <= j <= pos or j < keep, but none in (skip, next).  (Those that the products had already
// brought may be added once more: an infinity or NaN stays what it is.)  turned: the columns are pairs turned by an angle, and
// both become NaN.
template <typename T>
__device__ __noinline__ void add_odd_values(T* dst, const bf16* values, const int* table, int value_row, int KVH, int kvh, int page,
                                            int first, int skip, int next, int pos, int lo, int keep, int c0, int n, int half, bool turned) {
  for (int j = first; j <= pos; ++j) {
    if (j > skip && j < next) {
      j = next;
      if (j > pos) break;
    }
    if (j < lo && j >= keep) continue;
    const bf16* v = values + ((size_t)(table[j / page] * KVH + kvh) * page + j % page) * value_row;
    for (int c = c0; c < c0 + n; ++c) {
      const float x = to_f(v[c]), y = to_f(v[c + half]);
      const bool bad_x = !isfinite(x), bad_y = !isfinite(y);
      if (turned && (bad_x || bad_y)) {
        dst[c] = dst[c + half] = from_f<T>(NAN);
        continue;
      }
      if (bad_x) dst[c] = from_f<T>(to_f(dst[c]) + x);
      if (bad_y) dst[c + half] = from_f<T>(to_f(dst[c + half]) + y);
    }
  }
}

// The lowest n bits (n < 0: none; n > 31: all).
__device__ __forceinline__ uint32_t below(int n) { return n <= 0 ? 0u : (n >= 32 ? 0xffffffffu : (1u << n) - 1u); }

template <int DK, int DV, int TK, bool V_IN_K, int QT, bool MAPS = false>
__global__ void __launch_bounds__(THREADS, 1)
attention_biased_tc_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                           const __grid_constant__ CUtensorMap k_run_map, const __grid_constant__ CUtensorMap v_run_map,
                           const Args a) {
  using PL = Plan<DK, DV, TK, V_IN_K, QT, MAPS>;
  constexpr int KB = PL::KB, VB = PL::VB, STAGES = PL::STAGES, KT = PL::KT, UNITS = PL::UNITS;
  constexpr uint32_t BLK_KV = PL::BLK_KV;
  constexpr uint32_t K_BYTES = PL::K_BYTES, V_BYTES = PL::V_BYTES, S_COL = PL::S_COL, O_COL = PL::O_COL, Q_COL = PL::Q_COL;
  pdl_launch_dependents();
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* q_s = smem;                               // [KB - QT][128][128 B]
  unsigned char* k_s = q_s + PL::Q_BYTES;                  // [STAGES][KB][TK][128 B]
  unsigned char* v_s = k_s + STAGES * K_BYTES;             // [STAGES][VB][TK][128 B] (absent when the values are in the key rows)
  // (values in the key rows: the _k barriers are those of a tile's blocks that are no values here, the _v ones those of its values)
  uint64_t* full_k = reinterpret_cast<uint64_t*>(v_s + STAGES * V_BYTES);
  uint64_t* empty_k = full_k + STAGES;
  uint64_t* full_v = empty_k + STAGES;
  uint64_t* empty_v = full_v + STAGES;
  uint64_t* bar_s = empty_v + STAGES;                      // [2] S in that buffer is complete
  uint64_t* bar_p = bar_s + 2;                             // [2] all rows have consumed S(t) and written P(t)
  uint64_t* bar_pv = bar_p + 2;                            // an O product is complete
  uint64_t* bar_o = bar_pv + 1;                            // the last O product is complete
  uint64_t* bar_q = bar_o + 1;                             // the query rows are in place
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_k + (PL::BARRIERS + 1) / 2 * 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* odd_flag = abort_flag + 1;                 // a tile held infinities or NaN that not all rows may see
  float* max_x = reinterpret_cast<float*>(tmem_slot + 4);  // [tile & 1][2 halves][128 rows]

  // (two score maps a head, MAPS: a key row is [map 0 | map 1], a query [map 0 | map 1] too; a block takes one of them)
  const int b = blockIdx.z, kvh = MAPS ? blockIdx.y >> 1 : blockIdx.y, map_col = MAPS ? (blockIdx.y & 1) * DK : 0;
  const int chunk = blockIdx.x % a.v_chunks, tile = blockIdx.x / a.v_chunks;
  const int G = a.H / a.KVH;
  const int qs = a.q_start[b];
  const int q_len = a.q_start[b + 1] - qs;
  const int seq_len = a.seq_lens[b];
  const int n_rows = q_len * G;
  const int n_row_tiles = (n_rows + TQ - 1) / TQ;
  if (tile >= n_row_tiles || n_rows <= a.min_rows) return;
  const int row0 = (n_row_tiles - 1 - tile) * TQ;          // longest tiles first
  const int tid = threadIdx.x, warp = tid >> 5;
  const int prefix = seq_len - q_len;

  if ((smem_u32(smem) & 1023u) != 0) {                     // the swizzled tiles need 1024-byte alignment
    if (tid == 0) atomicCAS(a.status, 0, 9);
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_k[s], 1);
      mbar_init(&empty_k[s], 1);
      mbar_init(&full_v[s], 1);
      mbar_init(&empty_v[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_s[i], 1);
      mbar_init(&bar_p[i], SOFTMAX_THREADS);
    }
    mbar_init(bar_pv, 1);
    mbar_init(bar_o, 1);
    mbar_init(bar_q, SOFTMAX_THREADS);
    *abort_flag = 0;
    *odd_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(PL::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // The keys any row of the block can see: [j_first, j_hi] and, ahead of what a window shows, the kept first tokens (tiles
  // of their own).  j_lo: j_first aligned down to a TMA box.
  const int last_row = min(row0 + TQ, n_rows) - 1;
  const int j_hi = prefix + last_row / G;
  int j_first = a.window > 0 ? max(0, prefix + row0 / G - a.window + 1) : 0;
  if (a.block_of > 0) j_first = max(j_first, (prefix + row0 / G) / a.block_of * a.block_of);
  const int box = a.box;
  const int j_lo = j_first & ~(box - 1);
  const int keep_end = a.keep > 0 ? min(a.keep, j_lo) : 0;
  const int kept = (keep_end + TK - 1) / TK;
  // Keys [lo_all, hi_all] are seen by every row (its last row sees the fewest from below, its first from above); of those outside
  // them [j_first, j_hi] are seen by some.
  const int hi_all = prefix + row0 / G;
  int lo_all = a.window > 0 ? max(0, j_hi - a.window + 1) : 0;
  if (a.block_of > 0) lo_all = max(lo_all, j_hi / a.block_of * a.block_of);
  const int n_tiles = (seq_len > 0 && j_hi >= j_lo) ? kept + (j_hi - j_lo) / TK + 1 : 0;
  // Tiles are taken from the last to the first: with a bias that falls with the distance, and mostly without one, a row's
  // largest score comes early, and the reference that its exponentials refer to then stays where it is.
  auto tile_key = [&](int t) {
    const int u = n_tiles - 1 - t;
    return u < kept ? u * TK : j_lo + (u - kept) * TK;
  };

  // a softmax thread's row and which half of a tile's keys (and of the value columns) it takes
  const int lane_row = tid & (TQ - 1), hh = (tid >> 7) & 1;
  const int row = row0 + lane_row;
  const bool row_ok = tid < SOFTMAX_THREADS && row < n_rows;
  const int tok = row_ok ? row / G : 0, g = row_ok ? row % G : 0;
  const int pos = row_ok ? prefix + tok : -1;
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;

  pdl_wait();                                              // queries, keys and values of this step are written by earlier kernels

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp >= LOAD_WARP) {
    // ================= TMA loads, one lane of each of two warps: keys and values, or half of a latent tile each =================
    if ((tid & 31) == 0 && n_tiles > 0) {
      const bool first = warp == LOAD_WARP;
      // its 64-column blocks of a row: `count` of them from c0 on (values in the key rows: the first warp's step over them)
      const int count = first ? (V_IN_K ? KB - VB : KB) : VB;
      const int v0 = chunk * VB;
      auto block = [&](int i) { return V_IN_K ? (first ? (i < v0 ? i : i + VB) : v0 + i) : i; };
      const int col0 = V_IN_K ? 0 : (first ? map_col : chunk * DV);   // (the first column the block wants of a row)
      const CUtensorMap* map = V_IN_K || first ? &k_map : &v_map;
      const CUtensorMap* rmap = V_IN_K || first ? &k_run_map : &v_run_map;
      unsigned char* ring = V_IN_K || first ? k_s : v_s;
      uint64_t* full = first ? full_k : full_v;
      uint64_t* empty = first ? empty_k : empty_v;
      const uint32_t stage_bytes = V_IN_K || first ? K_BYTES : V_BYTES;
      const uint32_t mine = (uint32_t)count * BLK_KV;
      // The page ids of a tile whose pages are shorter than the tile (2 or 4 of them), read two tiles ahead: a table entry
      // fetched where it is used would put a trip to memory into every tile of the one thread that issues the copies.
      struct TilePages { int p[4 * UNITS]; };
      const int run = a.run;
      const int* tab_row = a.block_tables + (size_t)b * a.table_width;
      auto pages_of = [&](int t) {
        TilePages tp;
#pragma unroll
        for (int w = 0; w < UNITS; ++w) {
          const int lp0 = t < n_tiles ? (tile_key(t) + w * UNIT) / a.page : 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) tp.p[4 * w + i] = (i < run && t < n_tiles && lp0 + i < a.table_width) ? tab_row[lp0 + i] : -1;
        }
        return tp;
      };
      bool ok = true;
      TilePages cur = pages_of(0), nxt = pages_of(1);
      for (int t = 0; t < n_tiles && ok; ++t) {
        const TilePages after = pages_of(t + 2);
        const int st = t % STAGES;
        if (t >= STAGES) ok = mbar_wait(&empty[st], (uint32_t)((t / STAGES - 1) & 1), a.status, first ? 4 : 7, abort_flag);
        if (!ok) break;
        mbar_expect_tx(&full[st], mine);
#pragma unroll
        for (int w = 0; w < UNITS; ++w) {
          unsigned char* dst = ring + st * stage_bytes + w * UNIT * 128;
          const int j0 = tile_key(t) + w * UNIT;
          const int* pg = cur.p + 4 * w;
          bool in_a_row = run > 1 && pg[0] >= 0;
#pragma unroll
          for (int i = 1; i < 4; ++i) in_a_row = in_a_row && (i >= run || pg[i] == pg[0] + i);
          if (in_a_row) {
            // pages that follow one another in the pool: one box brings the unit's rows of 64 columns
            for (int c = 0; c < count; ++c) tma_load_run(dst + block(c) * BLK_KV, rmap, col0 + block(c) * 64, kvh, pg[0], &full[st]);
          } else if (run > 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (i >= run) break;
              const int y = (max(pg[i], 0) * a.KVH + kvh) * a.page;
              for (int c = 0; c < count; ++c) tma_load_2d(dst + block(c) * BLK_KV + i * a.page * 128, map, col0 + block(c) * 64, y, &full[st]);
            }
          } else {
            for (int bx = 0; bx < UNIT / box; ++bx) {
              const int j = j0 + bx * box;
              const int lp = j / a.page;
              const int page = lp < a.table_width ? tab_row[lp] : 0;
              const int y = (page * a.KVH + kvh) * a.page + (j - lp * a.page);
              for (int c = 0; c < count; ++c) tma_load_2d(dst + block(c) * BLK_KV + bx * box * 128, map, col0 + block(c) * 64, y, &full[st]);
            }
          }
        }
        cur = nxt;
        nxt = after;
      }
    }
  } else if (warp == MMA_WARP) {
    // ================= product issue, one lane =================
    if ((tid & 31) == 0 && n_tiles > 0) {
      // S(t) = Q . K(t)^T into buffer t & 1.  Everything but the stage is known at compile time (the chunk by the branch in
      // `scores`): one thread issues a product of 46 to 64 cycles, and building descriptors at run time took it longer.
      const uint64_t q_desc = smem_desc(smem_u32(q_s));
      auto products_s = [&](int t, auto from, auto to, auto start) {
        constexpr uint32_t idesc = instr_desc(TK);
        const uint64_t k_desc = smem_desc(smem_u32(k_s + (t % STAGES) * K_BYTES));
        const uint32_t d = tmem + S_COL + (t & 1) * TK;
#pragma unroll
        for (int blk = decltype(from)::value; blk < decltype(to)::value; ++blk) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint64_t kd = k_desc + ((blk * BLK_KV + ks * 32) >> 4);
            const uint32_t add = (decltype(start)::value && blk == decltype(from)::value && ks == 0) ? 0u : 1u;
            if (blk < QT) umma_ts(d, tmem + Q_COL + blk * 32 + ks * 8, kd, idesc, add);
            else umma(d, q_desc + (((blk - QT) * BLK_Q + ks * 32) >> 4), kd, idesc, add);
          }
        }
      };
      // O += (hi + lo)(t) . V(t), 16 keys (8 columns of bfloat16 pairs) at a time; V is MN-major as TMA left it
      auto products_o = [&](int t) {
        constexpr uint32_t idesc = instr_desc(DV, true);
        const uint32_t va = V_IN_K ? smem_u32(k_s + (t % STAGES) * K_BYTES) + chunk * VB * BLK_KV : smem_u32(v_s + (t % STAGES) * V_BYTES);
        const uint64_t v_desc = smem_desc_mn(va, BLK_KV);
        const uint32_t p = tmem + S_COL + (t & 1) * TK;
#pragma unroll
        for (int kk = 0; kk < TK / 16; ++kk) {
          const uint64_t vd = v_desc + (kk * 16 * 128 >> 4);
          const uint32_t hi = p + kk / (KT / 16) * KT + kk % (KT / 16) * 8;
          umma_ts(tmem + O_COL, hi, vd, idesc, (t > 0 || kk > 0) ? 1u : 0u);
          umma_ts(tmem + O_COL, hi + KT / 2, vd, idesc, 1u);
        }
        umma_commit(&empty_v[t % STAGES]);
        umma_commit(bar_pv);
        if (t + 1 == n_tiles) umma_commit(bar_o);
      };
      bool ok = mbar_wait(bar_q, 0, a.status, 11, abort_flag);
      auto scores = [&](int t) {
        const uint32_t parity = (uint32_t)((t / STAGES) & 1);
        ok = ok && mbar_wait(&full_k[t % STAGES], parity, a.status, 1, abort_flag);
        if (!ok) return;
        tc_fence_after();
        if constexpr (V_IN_K) {
          // the blocks that are no values here, then the values
          auto in_chunk = [&](auto c) {
            constexpr int v0 = decltype(c)::value * VB, v1 = v0 + VB;
            products_s(t, Int<0>{}, Int<v0>{}, Int<1>{});
            products_s(t, Int<v1>{}, Int<KB>{}, Int<(v0 == 0)>{});
            ok = mbar_wait(&full_v[t % STAGES], parity, a.status, 8, abort_flag);
            if (!ok) return;
            tc_fence_after();
            products_s(t, Int<v0>{}, Int<v1>{}, Int<0>{});
          };
          if (KB < 2 * VB || chunk == 0) in_chunk(Int<0>{});
          else in_chunk(Int<(KB < 2 * VB ? 0 : 1)>{});
          if (!ok) return;
        } else {
          products_s(t, Int<0>{}, Int<KB>{}, Int<1>{});
        }
        umma_commit(&bar_s[t & 1]);
        umma_commit(&empty_k[t % STAGES]);
      };
      auto outputs = [&](int t) {
        ok = ok && mbar_wait_spin(&bar_p[t & 1], (uint32_t)((t >> 1) & 1), a.status, 6, abort_flag);       // P(t) is in place
        if (!V_IN_K) ok = ok && mbar_wait(&full_v[t % STAGES], (uint32_t)((t / STAGES) & 1), a.status, 3, abort_flag);
        if (!ok) return;
        tc_fence_after();
        products_o(t);
      };
      for (int t = 0; t < 2 && t < n_tiles; ++t) scores(t);
      for (int t = 0; t < n_tiles && ok; ++t) {
        outputs(t);
        if (t + 2 < n_tiles) scores(t + 2);                // over P(t), behind the product that reads it
      }
    }
  } else {
    // ================= softmax warps: two threads per row = tensor-memory lane =================
    // Query rows: 64-column blocks 0 .. QT - 1 -> tensor memory (lane = row, a 32-bit column = two neighbouring query columns),
    // the others -> shared memory, K-major with the 128-byte swizzle (16-byte chunk c of row r at c ^ (r & 7)); of a row's two
    // threads each takes every second block
    const bf16* src = a.q + (size_t)(qs + tok) * a.q_ts + (size_t)(kvh * G + g) * a.q_hs + map_col;
#pragma unroll 1
    for (int blk = hh; blk < KB; blk += 2) {
      uint32_t w[32];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint4 v = row_ok ? *reinterpret_cast<const uint4*>(src + blk * 64 + c * 8) : make_uint4(0u, 0u, 0u, 0u);
        w[4 * c] = v.x;
        w[4 * c + 1] = v.y;
        w[4 * c + 2] = v.z;
        w[4 * c + 3] = v.w;
      }
      if (QT > 0 && blk < QT) {
        tmem_st32(tmem + lane_addr + Q_COL + blk * 32, w);
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(q_s + (blk - QT) * BLK_Q + lane_row * 128 + ((c ^ (lane_row & 7)) << 4)) =
              make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
      }
    }
    if (QT > 0) tmem_wait_st();
    fence_async_smem();
    tc_fence_before();
    mbar_arrive(bar_q);

    float m_ref = -INFINITY, l_run = 0.f;                  // the maximum the exponentials refer to; this half's sum in its scale
    const float sc = a.scale * LOG2E_F;
    const float slope = (a.slopes != nullptr && row_ok) ? a.slopes[kvh * G + g] * LOG2E_F : 0.f;      // (exp2 domain)
    const bool straight = a.softcap <= 0.f && a.slopes == nullptr && sc > 0.f;    // then the scale joins the exponential's argument
    const float mul = straight ? sc : 1.f;
    const float c_cap = a.softcap > 0.f ? a.softcap * LOG2E_F : 0.f, c_in = a.softcap > 0.f ? 2.f * sc / a.softcap : 0.f;
    int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;                // the first key the row sees (but for the kept ones)
    if (a.block_of > 0) lo = max(lo, max(pos, 0) / a.block_of * a.block_of);
    const int pair = warp & 3;                             // warps `pair` and `pair + 4` share 32 rows and barrier 1 + pair
    // The barrier of the two warps.  One that gives up on a wait of its own arrives without waiting (below), having set the
    // flag that the other then sees here, so that neither waits for good.
    auto meet = [&]() {
      asm volatile("bar.sync %0, 64;" ::"r"(1 + pair) : "memory");
      return __all_sync(0xffffffffu, *abort_flag == 0);
    };
    bool ok = true;
    for (int t = 0; t < n_tiles; ++t) {
      const uint32_t s_addr = tmem + lane_addr + S_COL + (t & 1) * TK;
      const int jt = tile_key(t);
      const int u = n_tiles - 1 - t;
      const int j_end = u < kept ? keep_end - 1 : j_hi;
      ok = mbar_wait(&bar_s[t & 1], (uint32_t)((t >> 1) & 1), a.status, 2, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      // Value rows of keys the block must not see are cleared (the first and the last tile of a stretch of keys only); what is
      // not finite among those that only some of its rows see is taken out.  (The kept first tokens are seen by all.)
      const bool partial = u >= kept && ((hi_all < j_hi && jt + TK - 1 > hi_all) || (lo_all > j_first && jt < lo_all));
      if (partial || jt + TK - 1 > j_end || (u == kept && jt < j_first)) {
        unsigned char* vt = V_IN_K ? k_s + (t % STAGES) * K_BYTES + chunk * VB * BLK_KV : v_s + (t % STAGES) * V_BYTES;
        ok = mbar_wait_spin(&full_v[t % STAGES], (uint32_t)((t / STAGES) & 1), a.status, 14, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        auto place = [&](int i) { return reinterpret_cast<uint4*>(vt + (i % (VB * 8) >> 3) * BLK_KV + i / (VB * 8) * 128 + (i & 7) * 16); };
        auto unseen = [&](int j) { return j > j_end || (j < j_first && u >= kept && j >= a.keep); };
        uint32_t some = 0;
        if (partial) {                                     // (all loads in flight: this is the common case, and nothing is found)
          uint4 v[TK * VB * 8 / SOFTMAX_THREADS];
#pragma unroll
          for (int k = 0; k < TK * VB * 8 / SOFTMAX_THREADS; ++k) v[k] = *place(tid + k * SOFTMAX_THREADS);
#pragma unroll
          for (int k = 0; k < TK * VB * 8 / SOFTMAX_THREADS; ++k) some |= odd(v[k].x) | odd(v[k].y) | odd(v[k].z) | odd(v[k].w);
        }
        if (some != 0) {
          for (int i = tid; i < TK * VB * 8; i += SOFTMAX_THREADS) {
            uint4* at = place(i);
            const uint4 v = *at;
            if (unseen(jt + i / (VB * 8)) || !(odd(v.x) | odd(v.y) | odd(v.z) | odd(v.w))) continue;
            *at = make_uint4(without_odd(v.x), without_odd(v.y), without_odd(v.z), without_odd(v.w));
            *odd_flag = 1;
          }
        }
        if (jt + TK - 1 > j_end || (u == kept && jt < j_first)) {
          for (int i = tid; i < TK * VB * 8; i += SOFTMAX_THREADS)
            if (unseen(jt + i / (VB * 8))) *place(i) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_async_smem();                                // (before this thread's arrival for P(t), which the product waits for)
      }
      const int j0 = jt + hh * KT;                         // this thread's first key of the tile
      // keys that every row of the warp sees (the common case away from the edges) need no mask (nor do rows that do not
      // exist: they store nothing)
      const bool all_visible = __all_sync(0xffffffffu, !row_ok || (j0 + KT - 1 <= min(pos, j_end) && (j0 >= lo || j0 + KT - 1 < a.keep)));
      uint32_t sv[KT];                                     // scores (times `mul`: in the exp2 domain), then the weights
      auto load_scores = [&]() {
#pragma unroll
        for (int h = 0; h < KT / 32; ++h) tmem_ld32(s_addr + hh * KT + h * 32, reinterpret_cast<uint32_t(&)[32]>(sv[h * 32]));
        tmem_wait_ld();
        if (!straight) {
          const float base = c_cap - slope * (float)(pos - j0);
#pragma unroll
          for (int i = 0; i < KT; ++i) {
            // cap tanh(x / cap) = cap - 2 cap / (e^(2 x / cap) + 1); the bias beside it
            const float bias = fmaf(slope, (float)i, base);
            const float v = __uint_as_float(sv[i]);
            sv[i] = __float_as_uint(a.softcap > 0.f ? fmaf(__fdividef(1.f, ex2(v * c_in) + 1.f), -2.f * c_cap, bias) : fmaf(v, sc, bias));
          }
        }
        if (!all_visible) {
          // bit i: key j0 + i is at most min(pos, j_end), and at least lo or below keep
#pragma unroll
          for (int h = 0; h < KT / 32; ++h) {
            const int jh = j0 + h * 32;
            const uint32_t vis = below(min(pos, j_end) + 1 - jh) & (~below(lo - jh) | below(a.keep - jh));
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (!(vis & (1u << i))) sv[h * 32 + i] = __float_as_uint(-INFINITY);
          }
        }
      };
      load_scores();
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < KT; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(sv[i]));
      float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * mul;
      // the row's maximum over both halves, as both threads must see the same one
      float* mx_s = max_x + (t & 1) * 2 * TQ + lane_row;   // (two tiles' places: the other thread may still read the last one)
      mx_s[hh * TQ] = mx;
      // the weights of this thread's keys as two bfloat16 terms, in pairs: hi in the first KT / 2 words, lo behind them
      auto exponentials = [&](float m_use) {
        float rs[2] = {0.f, 0.f};
        uint32_t lw[KT / 2];
#pragma unroll
        for (int i = 0; i < KT / 2; ++i) {
          const float p0 = ex2(fmaf(__uint_as_float(sv[2 * i]), mul, -m_use));
          const float p1 = ex2(fmaf(__uint_as_float(sv[2 * i + 1]), mul, -m_use));
          rs[i & 1] += p0 + p1;
          const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
          sv[i] = *reinterpret_cast<const uint32_t*>(&h2);
          const __nv_bfloat162 l2 = __floats2bfloat162_rn(p0 - __uint_as_float(sv[i] << 16), p1 - __uint_as_float(sv[i] & 0xffff0000u));
          lw[i] = *reinterpret_cast<const uint32_t*>(&l2);
        }
#pragma unroll
        for (int i = 0; i < KT / 2; ++i)
          sv[KT / 2 + i] = lw[i];
        return rs[0] + rs[1];
      };
      // The reference moves rarely once a row has one: the exponentials are taken against the present one while the other
      // thread's maximum is on its way, and taken again, from the scores in tensor memory, where one then moves after all.
      const bool ahead = __all_sync(0xffffffffu, m_ref != -INFINITY);
      float rs = 0.f;
      if (ahead) rs = exponentials(m_ref);
      ok = meet();
      if (!ok) break;
      mx = fmaxf(mx, mx_s[(hh ^ 1) * TQ]);
      const bool move = mx > m_ref + RESCALE_STEP || (m_ref == -INFINITY && mx > -INFINITY);
      float corr = 1.f;
      if (move) {
        corr = ex2(m_ref - mx);                            // 0 when there was no reference yet: O and l are 0 then
        m_ref = mx;
      }
      const bool any_move = __any_sync(0xffffffffu, move);
      if (!ahead || any_move) {
        if (ahead) load_scores();
        rs = exponentials((m_ref == -INFINITY) ? 0.f : m_ref);
      }
      l_run = l_run * corr + rs;
      // rescale O where a reference moved, each thread its half of the columns: the product before must be done with O
      if (t > 0 && any_move) {
        ok = mbar_wait_spin(bar_pv, (uint32_t)((t - 1) & 1), a.status, 10, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = hh * (DV / 2); c < (hh + 1) * (DV / 2); c += 32) {
          uint32_t ov[32];
          tmem_ld32(tmem + lane_addr + O_COL + c, ov);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
          tmem_st32(tmem + lane_addr + O_COL + c, ov);
        }
      }
#pragma unroll
      for (int h = 0; h < KT / 32; ++h)                    // over this thread's own scores
        tmem_st32(s_addr + hh * KT + h * 32, reinterpret_cast<uint32_t(&)[32]>(sv[h * 32]));
      tmem_wait_st();                                      // P (and a rescaled O) are in tensor memory
      tc_fence_before();
      mbar_arrive(&bar_p[t & 1]);
    }
    if (ok && n_tiles > 0) {
      ok = mbar_wait(bar_o, 0, a.status, 5, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (!ok) {
      __threadfence_block();
      asm volatile("bar.arrive %0, 64;" ::"r"(1 + pair) : "memory");
    } else if (n_tiles > 0) {
      // the row's sum is the two halves' sums (same scale), exchanged like the maxima
      float* l_s = max_x + (n_tiles & 1) * 2 * TQ + lane_row;
      l_s[hh * TQ] = l_run;
      ok = meet();
      if (ok) l_run += l_s[(hh ^ 1) * TQ];
    }
    if (ok) {
      tc_fence_after();
      const int head = kvh * G + g;
      float inv = 0.f;
      if (l_run > 0.f) {
        // the sink joins the denominator; both against the larger of the reference and the sink
        const float sink = a.sinks != nullptr ? a.sinks[head] * LOG2E_F : -INFINITY;
        const float top = fmaxf(m_ref, sink);
        const float down = exp2f(m_ref - top);
        inv = down / (l_run * down + exp2f(sink - top));
      }
      if (row_ok && a.fin.gate != nullptr)
        inv *= 1.f / (1.f + expf(-to_f(((const bf16*)a.fin.gate)[(size_t)(qs + tok) * a.fin.gate_ts + head])));
      bf16* dst = a.out + (size_t)(qs + tok) * a.out_ts + (size_t)head * a.out_hs + chunk * DV;
      // 16 columns and the 16 half a row further (so that pairs can be turned) at a time; each thread half of those
#pragma unroll 1
      for (int c = hh * (DV / 4); c < (hh + 1) * (DV / 4); c += 16) {
        uint32_t x[16], y[16];
        if (n_tiles > 0) {
          tmem_ld16(tmem + lane_addr + O_COL + c, x);      // the whole warp loads; rows without a query store nothing
          tmem_ld16(tmem + lane_addr + O_COL + DV / 2 + c, y);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = y[i] = 0u;
        }
        if (!row_ok) continue;
        if (MAPS) {
          float* dst32 = a.out32 + (size_t)(qs + tok) * a.out_ts + (size_t)head * a.out_hs + (MAPS && map_col ? DV : 0);
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            *reinterpret_cast<float4*>(dst32 + c + i) = make_float4(__uint_as_float(x[i]) * inv, __uint_as_float(x[i + 1]) * inv,
                                                                    __uint_as_float(x[i + 2]) * inv, __uint_as_float(x[i + 3]) * inv);
            *reinterpret_cast<float4*>(dst32 + DV / 2 + c + i) = make_float4(__uint_as_float(y[i]) * inv, __uint_as_float(y[i + 1]) * inv,
                                                                             __uint_as_float(y[i + 2]) * inv, __uint_as_float(y[i + 3]) * inv);
          }
          continue;
        }
        if (a.fin.out_freq != nullptr) {                   // (whole value rows only)
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float sn, cs;
            sincosf((float)pos * a.fin.out_freq[c + i], &sn, &cs);
            const float u = __uint_as_float(x[i]), w = __uint_as_float(y[i]);
            x[i] = __float_as_uint(u * cs + w * sn);
            y[i] = __float_as_uint(w * cs - u * sn);
          }
        }
#pragma unroll
        for (int i = 0; i < 16; i += 8) {
          uint32_t wx[4], wy[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 px = __floats2bfloat162_rn(__uint_as_float(x[i + 2 * e]) * inv, __uint_as_float(x[i + 2 * e + 1]) * inv);
            const __nv_bfloat162 py = __floats2bfloat162_rn(__uint_as_float(y[i + 2 * e]) * inv, __uint_as_float(y[i + 2 * e + 1]) * inv);
            wx[e] = *reinterpret_cast<const uint32_t*>(&px);
            wy[e] = *reinterpret_cast<const uint32_t*>(&py);
          }
          *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(wx[0], wx[1], wx[2], wx[3]);
          *reinterpret_cast<uint4*>(dst + DV / 2 + c + i) = make_uint4(wy[0], wy[1], wy[2], wy[3]);
        }
      }
      if (row_ok && *odd_flag) {
        const int skip = lo_all > j_first ? lo_all + TK - 2 : j_lo - 1, next = hi_all - TK + 2;
        const bf16* values = a.values + chunk * DV;
        const int* table = a.block_tables + (size_t)b * a.table_width;
        if (MAPS)
          add_odd_values(a.out32 + (size_t)(qs + tok) * a.out_ts + (size_t)head * a.out_hs + (map_col ? DV : 0), values, table, a.value_row,
                         a.KVH, kvh, a.page, j_lo, skip, next, pos, lo, a.keep, hh * (DV / 4), DV / 4, DV / 2, false);
        else
          add_odd_values(dst, values, table, a.value_row, a.KVH, kvh, a.page, j_lo, skip, next, pos, lo, a.keep, hh * (DV / 4), DV / 4, DV / 2,
                         a.fin.out_freq != nullptr);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PL::TMEM_COLS) : "memory");
  }
}

template <int DK, int DV, int TK, bool V_IN_K, int QT, bool MAPS = false>
int launch(dim3 grid, cudaStream_t stream, const CUtensorMap& k_map, const CUtensorMap& v_map, const CUtensorMap& k_run,
           const CUtensorMap& v_run, const Args& a) {
  using PL = Plan<DK, DV, TK, V_IN_K, QT, MAPS>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attention_biased_tc_kernel<DK, DV, TK, V_IN_K, QT, MAPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)PL::SMEM);
    if (e != cudaSuccess) TS_REFUSE((int)e, "ts_attention_biased_tc: shared memory %zu: %s", PL::SMEM, cudaGetErrorString(e));
    configured = true;
  }
  ts_launch(attention_biased_tc_kernel<DK, DV, TK, V_IN_K, QT, MAPS>, grid, dim3(THREADS), PL::SMEM, stream, k_map, v_map, k_run, v_run, a);
  TS_LAUNCH_CHECK();
}

// Two score maps a head (attention_diff.cu): every map of every kv head is a block's work like any other head's, with keys 64
// columns of the 128-wide key row.  The weights are two bfloat16 terms here too, although attention_diff_mma.cu has one: there the
// largest weight of a row is an exact 1, here it refers to a maximum that may lag behind, and with one term the outputs were
// up to 1.6 times further from 64 bits.  The two outputs stay in 32-bit until the kernel below has joined them.  2,048
// tokens, 12 heads over 2, the whole mixer: 193 us on mma.sync, 90 with one term, 99.7 with two.
// out[t, h] = out_scale * rms_norm(a_0 - lambda a_1) of the two maps' outputs, a warp a head; tokens of requests of min_rows
// rows or fewer are left alone.
template <int V>
__global__ void __launch_bounds__(128)
join_maps_kernel(bf16* __restrict__ out, const float* __restrict__ maps, const int* __restrict__ token_request,
                 const int* __restrict__ q_start, int H, int G, int min_rows, float lambda, float eps, float out_scale) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int PER = V / 32;
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int b = token_request[t];
  if (h >= H || (q_start[b + 1] - q_start[b]) * G <= min_rows) return;
  const float* src = maps + ((size_t)t * H + h) * 2 * V + lane * PER;
  float o[PER], ss = 0.f;
#pragma unroll
  for (int i = 0; i < PER; i += 2) {
    const float2 x = *reinterpret_cast<const float2*>(src + i), y = *reinterpret_cast<const float2*>(src + V + i);
    o[i] = x.x - lambda * y.x;
    o[i + 1] = x.y - lambda * y.y;
    ss = fmaf(o[i], o[i], fmaf(o[i + 1], o[i + 1], ss));
  }
  const float f = out_scale / sqrtf(warp_sum(ss) / (float)V + eps);
  bf16* dst = out + ((size_t)t * H + h) * V + lane * PER;
#pragma unroll
  for (int i = 0; i < PER; i += 2) *reinterpret_cast<__nv_bfloat162*>(dst + i) = __floats2bfloat162_rn(o[i] * f, o[i + 1] * f);
}

// which instance takes (key width, value width, values inside the key rows): 0 none
int instance_of(int Dk, int Dv, int v_in_k) {
  if (!v_in_k && Dk == 64 && Dv == 64) return 1;
  if (!v_in_k && Dk == 128 && Dv == 128) return 2;
  if (v_in_k && Dk == 576 && Dv == 512) return 3;
  if (v_in_k && Dk == 320 && Dv == 256) return 4;
  return 0;
}

}  // namespace

TS_API int ts_attention_biased_tc_supported(int H, int KVH, int Dk, int Dv, int v_in_k, int page, int dtype) {
  return dtype == TS_BF16 && KVH > 0 && H % KVH == 0 && page >= BOX_ROWS && page % BOX_ROWS == 0 && instance_of(Dk, Dv, v_in_k) != 0;
}

// As ts_attention_biased_mma without cut keys; num_pages: pages in the pools.  Refuses (TS_ERR_UNSUPPORTED) what the
// 16-byte accesses or the copies cannot take; that kernel then does.
TS_API int ts_attention_biased_tc(void* out, int out_ts, int out_hs, const void* q, int q_ts, int q_hs, const void* k_cache,
                                  const void* v_cache, const int* block_tables, const int* q_start, const int* seq_lens,
                                  int B, int table_width, int max_q_len, int H, int KVH, int Dk, int Dv, int page, int num_pages,
                                  float scale, float softcap, const float* slopes, int window, int block_of, const float* sinks,
                                  int keep, const float* out_freq, const void* gate, int gate_ts, void* stream) {
  if (B <= 0 || max_q_len <= 0) return 0;
  const int v_in_k = v_cache == nullptr;
  if (!ts_attention_biased_tc_supported(H, KVH, Dk, Dv, v_in_k, page, TS_BF16))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_biased_tc: H=%d KVH=%d keys %d values %d pages of %d", H, KVH, Dk, Dv, page);
  if ((q_ts % 8) || (q_hs % 8) || (out_ts % 8) || (out_hs % 8) || (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_biased_tc: rows must start on 16-byte boundaries");
  if (B > 65535 || KVH > 65535) TS_REFUSE(TS_ERR_LIMIT, "ts_attention_biased_tc: %d requests / %d kv heads", B, KVH);
  if (keep < 0 || (keep > 0 && block_of > 0)) TS_REFUSE(TS_ERR_SHAPE, "ts_attention_biased_tc: %d kept tokens (with blocks of %d)", keep, block_of);
  const int inst = instance_of(Dk, Dv, v_in_k);
  const int chunks = inst == 3 ? 2 : 1;
  if (out_freq != nullptr && chunks != 1)
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_biased_tc: values of %d are cut over blocks, their pairs cannot be turned", Dv);
  const long long rows = (long long)num_pages * KVH * page;
  if (num_pages <= 0 || rows > 0x7fffffffLL) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_biased_tc: cache of %lld rows", rows);
  int* status = ts_attn_status_word();
  if (status == nullptr) TS_REFUSE(TS_ERR_LIMIT, "ts_attention_biased_tc: no status word");
  const int box = page % 64 == 0 ? 64 : (page % 32 == 0 ? 32 : 16);
  const int run = (page < UNIT && box == page) ? UNIT / page : 0;
  CUtensorMap k_map, v_map, k_run, v_run;
  if (!tensor_map(&k_map, k_cache, (int)rows, Dk, box) || (!v_in_k && !tensor_map(&v_map, v_cache, (int)rows, Dv, box)))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_biased_tc: cuTensorMapEncodeTiled failed");
  if (v_in_k) v_map = k_map;
  k_run = k_map;
  v_run = v_map;
  if (run > 1 && (!run_map(&k_run, k_cache, num_pages, KVH, page, run, Dk) ||
                  (!v_in_k && !run_map(&v_run, v_cache, num_pages, KVH, page, run, Dv))))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_biased_tc: cuTensorMapEncodeTiled (runs of pages) failed");
  Args a;
  a.out = (bf16*)out;
  a.out32 = nullptr;
  a.min_rows = 0;
  a.q = (const bf16*)q;
  a.values = (const bf16*)(v_in_k ? k_cache : v_cache);
  a.value_row = v_in_k ? Dk : Dv;
  a.block_tables = block_tables;
  a.q_start = q_start;
  a.seq_lens = seq_lens;
  a.slopes = slopes;
  a.sinks = sinks;
  a.out_ts = out_ts;
  a.out_hs = out_hs;
  a.q_ts = q_ts;
  a.q_hs = q_hs;
  a.table_width = table_width;
  a.H = H;
  a.KVH = KVH;
  a.page = page;
  a.box = box;
  a.run = run > 1 ? run : 0;
  a.scale = scale;
  a.softcap = softcap;
  a.window = window;
  a.block_of = block_of;
  a.keep = keep;
  a.v_chunks = chunks;
  a.fin.out_freq = out_freq;
  a.fin.gate = gate;
  a.fin.gate_ts = gate_ts;
  a.status = status;
  dim3 grid(ceil_div(max_q_len * (H / KVH), TQ) * chunks, KVH, B);
  cudaStream_t s = (cudaStream_t)stream;
  if (inst == 1) return launch<64, 64, 128, false, 0>(grid, s, k_map, v_map, k_run, v_run, a);
  if (inst == 2) return launch<128, 128, 128, false, 0>(grid, s, k_map, v_map, k_run, v_run, a);
  if (inst == 3) return launch<576, 256, 64, true, 4>(grid, s, k_map, v_map, k_run, v_run, a);
  return launch<320, 256, 64, true, 0>(grid, s, k_map, v_map, k_run, v_run, a);
}

TS_API int ts_attention_maps_tc_supported(int H, int KVH, int D, int V, int page, int dtype) {
  return dtype == TS_BF16 && KVH > 0 && H % KVH == 0 && page >= BOX_ROWS && page % BOX_ROWS == 0 && D == 64 && (V == 64 || V == 128);
}

// Attention with two score maps a head (see attention_diff.cu) for the portions of more than min_rows query rows: maps [T, H, 2,
// V] 32-bit is work memory.  q: rows of proj, heads of 2 D; key rows of 2 D, value rows of V; out [T, H V].
TS_API int ts_attention_maps_tc(void* out, float* maps, const void* proj, int proj_stride, const void* k_cache, const void* v_cache,
                                const int* block_tables, const int* q_start, const int* seq_lens, const int* token_request, int B,
                                int T, int table_width, int max_q_len, int H, int KVH, int D, int V, int page, int num_pages,
                                float scale, float lambda, float eps, float out_scale, int min_rows, void* stream) {
  if (B <= 0 || max_q_len <= 0 || T <= 0) return 0;
  if (!ts_attention_maps_tc_supported(H, KVH, D, V, page, TS_BF16))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_maps_tc: H=%d KVH=%d maps of %d values %d pages of %d", H, KVH, D, V, page);
  if ((proj_stride % 8) || (((uintptr_t)proj | (uintptr_t)out | (uintptr_t)maps | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_maps_tc: rows must start on 16-byte boundaries");
  if (B > 65535 || KVH > 32767) TS_REFUSE(TS_ERR_LIMIT, "ts_attention_maps_tc: %d requests / %d kv heads", B, KVH);
  const long long rows = (long long)num_pages * KVH * page;
  if (num_pages <= 0 || rows > 0x7fffffffLL) TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_maps_tc: cache of %lld rows", rows);
  int* status = ts_attn_status_word();
  if (status == nullptr) TS_REFUSE(TS_ERR_LIMIT, "ts_attention_maps_tc: no status word");
  const int box = page % 64 == 0 ? 64 : (page % 32 == 0 ? 32 : 16);
  const int run = (page < UNIT && box == page) ? UNIT / page : 0;
  CUtensorMap k_map, v_map, k_run, v_run;
  if (!tensor_map(&k_map, k_cache, (int)rows, 2 * D, box) || !tensor_map(&v_map, v_cache, (int)rows, V, box))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_maps_tc: cuTensorMapEncodeTiled failed");
  k_run = k_map;
  v_run = v_map;
  if (run > 1 && (!run_map(&k_run, k_cache, num_pages, KVH, page, run, 2 * D) || !run_map(&v_run, v_cache, num_pages, KVH, page, run, V)))
    TS_REFUSE(TS_ERR_UNSUPPORTED, "ts_attention_maps_tc: cuTensorMapEncodeTiled (runs of pages) failed");
  Args a = {};
  a.out32 = maps;
  a.q = (const bf16*)proj;
  a.values = (const bf16*)v_cache;
  a.value_row = V;
  a.block_tables = block_tables;
  a.q_start = q_start;
  a.seq_lens = seq_lens;
  a.out_ts = H * 2 * V;
  a.out_hs = 2 * V;
  a.q_ts = proj_stride;
  a.q_hs = 2 * D;
  a.table_width = table_width;
  a.H = H;
  a.KVH = KVH;
  a.page = page;
  a.box = box;
  a.run = run > 1 ? run : 0;
  a.scale = scale;
  a.v_chunks = 1;
  a.min_rows = min_rows;
  a.status = status;
  const int G = H / KVH;
  const dim3 grid(ceil_div(max_q_len * G, TQ), 2 * KVH, B), join(T, ceil_div(H, 4));
  cudaStream_t s = (cudaStream_t)stream;
  int rc;
  if (V == 128) {
    rc = launch<64, 128, 128, false, 0, true>(grid, s, k_map, v_map, k_run, v_run, a);
    if (rc == 0)
      ts_launch(join_maps_kernel<128>, join, dim3(128), 0, s, (bf16*)out, maps, token_request, q_start, H, G, min_rows, lambda, eps, out_scale);
  } else {
    rc = launch<64, 64, 128, false, 0, true>(grid, s, k_map, v_map, k_run, v_run, a);
    if (rc == 0)
      ts_launch(join_maps_kernel<64>, join, dim3(128), 0, s, (bf16*)out, maps, token_request, q_start, H, G, min_rows, lambda, eps, out_scale);
  }
  if (rc != 0) return rc;
  TS_LAUNCH_CHECK();
}
