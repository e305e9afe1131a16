// Packed variable-length flash attention for sm_100a (forward + backward), GQA aware: causal
// inside each document, or bidirectional for documents whose tiles carry flag bit 0.
//
// Layout: tokens of all documents of a packed row are concatenated: q/k/v live in one fused
// projection buffer [T, (Hq + 2*Hk) * D] (bf16), documents are delimited by a host-built tile
// table (one entry per (document, 128-row tile)), so no [S,S] mask and no cross-document
// attention ever exists. Both kernels are warp-specialised:
//   warp 0: TMA producer, warp 1: tcgen05.mma issuer, two (forward) or four (backward) warpgroups: softmax / gradient math
// with S, P, O (forward) and S^T, dP^T, dK, dV, dQ^T (backward) accumulators living in TMEM.
//
// Replaces flash-attn varlen (FA2/FA4) that the reference reaches through HF's
// flash_attention_2 interface (src/axolotl/monkeypatch/attention/flash_attn_4.py:37-111) and its
// Triton varlen kernel (src/axolotl/monkeypatch/attention/flash_attn_d512.py:65-546).
#include "attn_common.cuh"
#include <type_traits>

namespace {

constexpr int HALF_BYTES = 128 * 128;  // 128 rows x 128 B (64 bf16) swizzled tile

struct AttnParams {
  const int4* tiles;  // (doc_start, doc_len, tile_start (doc relative), flags: bit 0 = bidirectional, bits 1.. = sliding window in tokens)
  int n_tiles;
  int Hq, Hk;
  int q_col0, k_col0, v_col0;  // element offsets of the q / k / v blocks inside a fused row
  __nv_bfloat16* out;          // [T, Hq*D]
  long long out_ld;
  float* lse2;  // [Hq, T]  log2-domain logsumexp of the scaled scores
  long long T;
  long long kv_rows;  // rows of the k / v buffer (the whole token stream under context parallelism)
  float sl2;  // softmax_scale * log2(e)
  int* status;
  // backward only
  const float* delta;  // [Hq, T]
  float* dq_acc;       // T * Hq * D fp32 in the order of dq_at, accumulated with reductions
  __nv_bfloat16* dkv;  // fused gradient buffer, same layout as qkv (k and v blocks are written)
  long long dkv_ld;
  float scale;
  // context parallelism: the q / out / lse / dO / dq buffers hold only the rows
  // [q_row_off, q_row_off + q_rows) of the global token stream, K and V are global.
  int q_row_off, q_rows;
  // backward with context parallelism: dK / dV tiles are reduce-added (bf16x2 atomics over
  // NVLink) into the buffer of the rank that owns the kv rows: rank = row / cp_chunk.
  int dk_col0, dv_col0;  // column offsets of the dK / dV blocks in the gradient buffer
  int cp_world;
  long long cp_chunk;
  unsigned long long cp_dkv_ptrs[8];
  // backward: the q heads of one kv head may be split over `kv_split` CTAs (load balance for wide
  // GQA groups); their dK / dV partial tiles are then reduce-added into a pre-zeroed buffer
  int kv_split;
  // forward: the two units of a CTA. 0: one unit, 1: two q heads of a kv head, 2: two neighbouring q tiles of a head
  int pair_mode;
};

// =====================================================================================
// Forward
// =====================================================================================
// A CTA works on two 128-row units of queries against one stream of K / V tiles: two q heads of the same kv head at the same
// rows (GQA groups of even size), or two neighbouring q tiles of one head. Each unit has its own softmax warpgroup and its own
// S and O in TMEM, [S0 | S1 | O0 | O1]; while one warpgroup exponentiates, the tensor core runs the other unit's P.V and next
// scores, and K / V are read once for both. P (bf16) overwrites the first half of its S columns and is the TMEM operand of
// P.V, so it never passes through shared memory. O accumulates in TMEM; a warp rescales its rows when one of them has a new
// maximum. Waiting until a maximum has grown by 2^8 would spare most of that (one 16384-token document 1.73 ms) and was taken
// back: with a reference below the maximum the largest P of a row is not exactly one, and rounding it to bf16 makes the error
// against 64 bits 1.5 % larger for unit normal q and k, 19 % for twice that. Dividing by the sum of the rounded P mends half.
// Bound: exponentials (16 per clock and SM against 1024 clocks of MMA per 128 x 128 block) and the MMA stream, about level.
// One 16384-token document, 32 / 8 heads of 128: 3.01 -> 1.89 ms (730 -> 1160 TFLOP/s) against one softmax warpgroup with O in
// registers and P through shared memory; 4 x 2048 268 -> 180 us; 11 x 707, 64 heads of 64, 279 -> 178 us. These are single calls with
// a cold L2; the long document takes 2.14 ms where calls follow one another and the board's power limit lowers the clock.
// TMA warp, MMA warp, two idle warps (they complete the warpgroup that gives registers away), 2 x 4 softmax warps. A row of S
// is held in 128 registers: the 384 x 168 registers of the launch are split 128 x 40 + 256 x 232.
constexpr int kFwdThreads = 384;
template <int D>
struct FwdCfg {
  static constexpr int HALVES = D / 64;
  static constexpr int TILE_BYTES = HALVES * HALF_BYTES;  // Q / K / V tile of 128 rows
  static constexpr int KV_STAGES = 2;
  static constexpr int SMEM = TILE_BYTES * (2 + 2 * KV_STAGES) + 1024 + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int O_COL = 256;    // O of unit u at O_COL + u * D; S (and P) of unit u at u * 128
};

template <int D>
__global__ void __launch_bounds__(kFwdThreads, 1)
    flash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_qkv,
                     const AttnParams p) {
  using C = FwdCfg<D>;
  const int tile_id = blockIdx.y;
  if (tile_id >= p.n_tiles) return;
  const int4 ti = p.tiles[tile_id];
  const int doc_start = ti.x, doc_len = ti.y, q0 = ti.z;
  if (!AXB_INDEX_OK(AXB_SITE_ATTN_TILE, (long long)doc_start + doc_len - 1, p.kv_rows) || !AXB_INDEX_OK(AXB_SITE_ATTN_TILE, q0, doc_len)) return;
  if (p.pair_mode == 2 && (q0 & 128)) return;   // the tile above takes these rows along
  const bool bidir = ti.w & 1;  // every token of the document sees the whole document
  const int win = bidir ? 0 : (ti.w >> 1);  // sliding window: row q sees kv rows (q - win, q]; 0 = unlimited
  const int head0 = p.pair_mode == 1 ? 2 * (int)blockIdx.x : (int)blockIdx.x;
  const int kv_head = head0 / (p.Hq / p.Hk);
  const int jb0 = win > 0 ? max(0, q0 - win + 1) / 128 : 0;  // first kv block any row of the first unit can see
  // kv blocks jb0 .. jb0 + n - 1 of a unit (0: no such unit)
  auto blocks_of = [&](int unit) -> int {
    if (unit == 1 && (p.pair_mode == 0 || (p.pair_mode == 2 && q0 + 128 >= doc_len))) return 0;
    const int top = p.pair_mode == 2 && unit == 1 ? q0 + 256 : q0 + 128;
    return ((bidir ? doc_len : min(top, doc_len)) + 127) / 128 - jb0;
  };
  const int n_u0 = blocks_of(0), n_u1 = blocks_of(1), n_max = max(n_u0, n_u1);
  // The window of the lower tile may begin a block later. Its P is zero in that block and is not multiplied by V, whose rows
  // there are none of its business (0 x inf is not 0).
  const int first_u1 = p.pair_mode == 2 && win > 0 ? max(0, q0 + 128 - win + 1) / 128 - jb0 : 0;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;                                // [2 units]
  uint8_t* sK = sQ + 2 * C::TILE_BYTES;
  uint8_t* sV = sK + C::KV_STAGES * C::TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + C::KV_STAGES * C::TILE_BYTES);
  uint64_t* q_full = bars + 0;    // [unit]
  uint64_t* k_full = bars + 2;    // [stage]
  uint64_t* v_full = bars + 4;    // [stage]
  uint64_t* k_empty = bars + 6;   // [stage]
  uint64_t* v_empty = bars + 8;   // [stage]
  uint64_t* s_full = bars + 10;   // [unit]  scores ready; every MMA issued before them has retired, P.V of the block before included
  uint64_t* p_full = bars + 12;   // [unit]  P written (S read, O rescaled)
  uint64_t* o_full = bars + 14;   // [unit]  O final
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 128);
      mbar_init(&o_full[s], 1);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tm_qkv);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
      auto load = [&](uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int col, int row) {
        if (elect_one()) {
          mbar_expect_tx(bar, C::TILE_BYTES);
#pragma unroll
          for (int h = 0; h < C::HALVES; ++h) tma_load_2d(dst + h * HALF_BYTES, m, bar, col + h * 64, row);
        }
        __syncwarp();
      };
      const int qrow = doc_start + q0 - p.q_row_off;
      load(sQ, &tm_q, &q_full[0], p.q_col0 + head0 * D, qrow);
      for (int j = 0; j < n_max; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        const int row = doc_start + (jb0 + j) * 128;
        if (!warp_all(mbar_wait(&k_empty[st], ph ^ 1, p.status, AXB_TIMEOUT_EMPTY))) break;
        load(sK + st * C::TILE_BYTES, &tm_qkv, &k_full[st], p.k_col0 + kv_head * D, row);
        if (j == 0 && n_u1 > 0)
          load(sQ + C::TILE_BYTES, &tm_q, &q_full[1], p.q_col0 + (p.pair_mode == 1 ? head0 + 1 : head0) * D,
               p.pair_mode == 2 ? qrow + 128 : qrow);
        if (!warp_all(mbar_wait(&v_empty[st], ph ^ 1, p.status, AXB_TIMEOUT_EMPTY))) break;
        load(sV + st * C::TILE_BYTES, &tm_qkv, &v_full[st], p.v_col0 + kv_head * D, row);
      }
    } else if (warp == 1) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);  // Q (K-major) x K (K-major)
      constexpr uint32_t idesc_pv = make_idesc_bf16(128, D, 0, 1);   // P (TMEM) x V (MN-major)
      const uint64_t dq_base = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), dk_base = make_smem_desc_sw128(smem_u32(sK), 16, 1024);
      const uint64_t dv_base = make_smem_desc_sw128(smem_u32(sV), HALF_BYTES, 1024);
      constexpr uint32_t TILE16 = C::TILE_BYTES / 16;
      auto issue_s = [&](int u, int j) {
        const uint64_t dq = dq_base + (uint32_t)u * TILE16, dk = dk_base + (uint32_t)(j & 1) * TILE16;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = ((kk / 4) * HALF_BYTES + (kk % 4) * 32) / 16;
            umma_f16(tmem_base + u * 128, dq + off, dk + off, idesc_s, kk > 0);
          }
          umma_commit(&s_full[u]);
        }
        __syncwarp();
      };
      auto issue_pv = [&](int u, int j, int first, bool last) {
        const uint64_t dv = dv_base + (uint32_t)(j & 1) * TILE16;
        if (j >= first && elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)   // 128 kv rows / 16: 8 TMEM columns of P each
            umma_f16_ts(tmem_base + C::O_COL + u * D, tmem_base + u * 128 + kk * 8, dv + kk * (2048 / 16), idesc_pv,
                        (j > first || kk > 0) ? 1u : 0u);
          if (last) umma_commit(&o_full[u]);
        }
        __syncwarp();
      };
      auto commit = [&](uint64_t* bar) {
        if (elect_one()) umma_commit(bar);
        __syncwarp();
      };
      bool ok = warp_all(mbar_wait(&q_full[0], 0, p.status, AXB_TIMEOUT_FULL) && mbar_wait(&k_full[0], 0, p.status, AXB_TIMEOUT_FULL));
      if (ok) {
        tc_fence_after();
        issue_s(0, 0);
        if (n_u1 > 0) {
          ok = warp_all(mbar_wait(&q_full[1], 0, p.status, AXB_TIMEOUT_FULL));
          if (ok) {
            tc_fence_after();
            issue_s(1, 0);
          }
        }
        commit(&k_empty[0]);
      }
      for (int j = 0; j < n_max && ok; ++j) {
        const int st = j & 1, nst = st ^ 1;
        bool v_ready = false, k_ready = false;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int n_u = u == 0 ? n_u0 : n_u1;
          if (j >= n_u || !ok) continue;
          ok = mbar_wait(&p_full[u], j & 1, p.status, AXB_TIMEOUT_GENERIC);
          if (ok && !v_ready) ok = mbar_wait(&v_full[st], (j >> 1) & 1, p.status, AXB_TIMEOUT_FULL);
          ok = warp_all(ok);
          if (!ok) break;
          v_ready = true;
          tc_fence_after();
          issue_pv(u, j, u == 0 ? 0 : first_u1, j == n_u - 1);
          if (j + 1 < n_u) {
            if (!k_ready) ok = warp_all(mbar_wait(&k_full[nst], ((j + 1) >> 1) & 1, p.status, AXB_TIMEOUT_FULL));
            if (!ok) break;
            k_ready = true;
            tc_fence_after();
            issue_s(u, j + 1);     // over P(j), which the P.V before it has read
          }
        }
        if (!ok) break;
        commit(&v_empty[st]);
        if (j + 1 < n_max) commit(&k_empty[nst]);
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax warpgroups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int u = (warp - 4) >> 2;
    const int lg = warp & 3;
    const int r = lg * 32 + lane;  // row inside the unit
    const int n_u = u == 0 ? n_u0 : n_u1;
    const int qu0 = p.pair_mode == 2 ? q0 + u * 128 : q0;
    const int head = p.pair_mode == 1 ? head0 + u : head0;
    const int q_idx = qu0 + r;
    const uint32_t lane_off = uint32_t(lg * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + u * 128, o_addr = tmem_base + lane_off + C::O_COL + u * D;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_u; ++j) {
      // A lane whose wait ran out walks on with the others, without waiting again: agreeing on every wait costs the chain 3 %
      // (one 16384-token document 1.89 -> 1.94 ms).
      ok = ok && mbar_wait(&s_full[u], j & 1, p.status, AXB_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      uint32_t sr[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, sr[c]);
      tmem_ld_wait();
      const int kv0 = (jb0 + j) * 128;
      if ((j == n_u - 1) || (win > 0 && kv0 < qu0 + 128 - win)) {
        const int lim = (bidir ? doc_len - 1 : min(q_idx, doc_len - 1)) - kv0;  // columns <= lim are visible
        const int lo = win > 0 ? q_idx - win + 1 - kv0 : -(1 << 30);            // columns >= lo are visible
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > lim || c * 32 + i < lo) sr[c][i] = 0xff800000u;    // -inf
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(sr[c][i]));
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.sl2);
      if (j == 0) {
        m = m_new;
      } else if (__any_sync(0xffffffffu, m_new > m)) {
        const float alpha = m_new == m ? 1.f : fast_exp2(m - m_new);
        m = m_new;
        l *= alpha;
#pragma unroll 1
        for (int c = 0; c < D / 64; ++c) {
          uint32_t o[2][32];
          tmem_ld_32x32(o_addr + c * 64, o[0]);
          tmem_ld_32x32(o_addr + c * 64 + 32, o[1]);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            o[0][i] = __float_as_uint(__uint_as_float(o[0][i]) * alpha);
            o[1][i] = __float_as_uint(__uint_as_float(o[1][i]) * alpha);
          }
          tmem_st_32x32(o_addr + c * 64, o[0]);
          tmem_st_32x32(o_addr + c * 64 + 32, o[1]);
        }
      }
      const float m_use = m == -INFINITY ? 0.f : m;    // no visible column so far: every P is exp2(-inf) = 0
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(sr[c][i]), p.sl2, -m_use));
          const float p1 = fast_exp2(fmaf(__uint_as_float(sr[c][i + 1]), p.sl2, -m_use));
          sum[i & 2] += p0;
          sum[(i & 2) + 1] += p1;
          pk[i >> 1] = pack_bf16x2(p0, p1);
        }
        tmem_st_32x16(s_addr + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[u]);
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
    if (warp_all(ok && n_u > 0 && mbar_wait(&o_full[u], 0, p.status, AXB_TIMEOUT_TMEM_FULL))) {
      tc_fence_after();
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      const long long lrow = (long long)doc_start + q_idx - p.q_row_off;  // row in the local buffers
      const bool row_ok = q_idx < doc_len && lrow >= 0 && lrow < p.q_rows;
      __nv_bfloat16* orow = p.out + lrow * p.out_ld + (long long)head * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(o_addr + c * 32, o);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(o[q * 8 + i]) * inv_l;
            *reinterpret_cast<uint4*>(orow + c * 32 + q * 8) =
                make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
        }
      }
      if (row_ok) p.lse2[(long long)head * p.q_rows + lrow] = m + log2f(l);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// =====================================================================================
// Backward
// =====================================================================================
// One CTA per (kv tile of 128 rows, kv head). Inner loop over the q heads of the GQA group and
// over 64-row q tiles at or below the diagonal. Every MMA has M = 128:
//   S^T  [kv, q]  = K . Q^T        dP^T [kv, q] = V . dO^T
//   dV   [kv, d] += P^T . dO       dK   [kv, d] += dS^T . Q
//   dQ^T [d,  q]  = K^T . dS^T     (drained with fp32 reductions into dq_acc)
// Two pairs of softmax warpgroups alternate iterations, each warpgroup with 32 of the 64 queries: S^T / dP^T (TMEM) and P^T / dS^T
// are double buffered, so the tensor core computes S^T, dP^T of iteration i+1 while pair i % 2 turns S^T(i) into P^T, dS^T and
// drains dQ^T(i). dQ^T(i) reuses the TMEM columns of S^T(i), which is dead once P^T(i) is written; with D = 128 all 512 columns are
// in use:
//   [S^T0 | dP^T0 | S^T1 | dP^T1 | dV (D) | dK (D)]
// What bounds it is the chain of a pair (scores -> P^T, dS^T -> dQ^T -> next scores); the tensor core is busy for 72 % of the time,
// 52 % without the operand reads (4 x 2048 tokens, 32 / 8 heads of 128: five products of 64 queries, three of them limited by the
// shared-memory reads of their 64 columns). 18 warps leave a thread 96 registers, of which heads of 128 spill nine. So nothing waits
// for memory inside the chain: Q / dO run three stages ahead (with two a quarter slower), lse and delta are requested two iterations
// early, dQ^T is the first product of its iteration and is drained while dV and dK run, and its sums leave by tile reductions: from
// registers they filled the load-store queue ahead of the other pair's dS^T (a fifth of the time). Whole backward pass (zeroing, delta,
// this kernel, conversion) against the form with two softmax warpgroups and single reductions, cold L2 / eight calls in turn: one
// 16384-token document, 32 / 8 heads of 128, 6.25 / 6.87 -> 5.18 / 5.99 ms; 4096 tokens, 32 / 4 heads of 64, 437 / 420 -> 330 / 314 us;
// 11 x 707 tokens, 64 / 8 heads of 64, window 128, 300 / 295 -> 287 / 279 (188 of them this kernel).
constexpr int kBwdThreads = 576;  // TMA warp, MMA warp, 4 x 4 softmax warps
template <int D>
struct BwdCfg {
  static constexpr int HALVES = D / 64;
  static constexpr int KV_BYTES = HALVES * HALF_BYTES;  // K or V tile: 128 rows
  static constexpr int Q_HALF = 64 * 128;               // 64 rows x 128 B
  static constexpr int Q_BYTES = HALVES * Q_HALF;       // Q or dO tile: 64 rows
  static constexpr int PT_BYTES = HALF_BYTES;           // P^T / dS^T: [128 kv x 64 q]
  // P^T as the TMEM operand of dV where shared memory is full; from shared memory is 1 to 3 % faster (whole backward pass, 32 / 4
  // heads of 64, 4096 tokens 292 against 295 us, 64 / 8 heads, 11 x 707 tokens 396 against 408; heads of 128 with P^T in shared memory
  // and two stages of Q / dO instead of three: a quarter slower)
  static constexpr bool PT_TMEM = D == 128;
  // dQ^T on its way out, per warp that owns rows of it: groups of four queries x 32 columns of d, all nine that 32 queries can touch
  // where shared memory allows
  static constexpr int OUT_GROUPS = D == 128 ? 4 : 8;      // rows of the tensor map's box
  static constexpr int OUT_BYTES = (D == 128 ? 4 : 9) * 512;
  static constexpr int STAGES = 3;                      // Q / dO: the load of a stage hides behind two iterations
  static constexpr int SMEM = 2 * KV_BYTES + STAGES * 2 * Q_BYTES + (PT_TMEM ? 2 : 4) * PT_BYTES + D / 8 * OUT_BYTES + 2048 /*lse+delta*/ + 256;
  static_assert(SMEM <= 227 * 1024, "");
  static constexpr int ST_COL = 0;     // S^T(b) at ST_COL + 128 b, 64 cols; dQ^T(b) aliases it
  static constexpr int DPT_COL = 64;   // dP^T(b) at DPT_COL + 128 b, 64 cols; P^T(b) (bf16) in the first half of each 32 (D = 128)
  static constexpr int DV_COL = 256;   // D cols
  static constexpr int DK_COL = 256 + D;
  static constexpr int TMEM_COLS = 512;
};

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
    flash_bwd_kernel(const __grid_constant__ CUtensorMap tm_kv,   // box 64 x 128 over qkv
                     const __grid_constant__ CUtensorMap tm_q,    // box 64 x 64 over qkv
                     const __grid_constant__ CUtensorMap tm_do,   // box 64 x 64 over dO
                     const __grid_constant__ CUtensorMap tm_dq,   // box OUT_GROUPS x 128 fp32 over dq_acc, a row per four queries
                     const AttnParams p) {
  using C = BwdCfg<D>;
  const int tile_id = blockIdx.y;
  if (tile_id >= p.n_tiles) return;
  const int kv_head = blockIdx.x / p.kv_split;
  const int part = blockIdx.x - kv_head * p.kv_split;
  const int group_all = p.Hq / p.Hk;
  const int group = group_all / p.kv_split;             // q heads handled by this CTA
  const int head0 = kv_head * group_all + part * group;  // first of them
  const int4 ti = p.tiles[tile_id];
  const int doc_start = ti.x, doc_len = ti.y, kv0 = ti.z;
  if (!AXB_INDEX_OK(AXB_SITE_ATTN_TILE, (long long)doc_start + doc_len - 1, p.kv_rows) || !AXB_INDEX_OK(AXB_SITE_ATTN_TILE, kv0, doc_len)) return;
  const bool bidir = ti.w & 1;
  // 64-row q tiles at or below the diagonal (all of the document's when it is bidirectional)
  // that intersect this rank's q rows
  const int win = bidir ? 0 : (ti.w >> 1);  // sliding window (0 = unlimited): kv row c is seen by q rows [c, c + win)
  int q_first = bidir ? 0 : kv0 / 64;
  int q_last = (doc_len + 63) / 64;
  if (win > 0) q_last = min(q_last, (kv0 + 127 + win - 1) / 64 + 1);
  {
    const int lo = p.q_row_off - doc_start, hi = p.q_row_off + p.q_rows - doc_start;
    if (lo > 0) q_first = max(q_first, lo / 64);
    q_last = min(q_last, (hi + 63) / 64);
  }
  const int n_qt = q_last - q_first;  // q tiles per head
  const int n_iter = n_qt * group;
  if (n_iter <= 0) return;

  // Every swizzled tile and descriptor needs a 1024-byte boundary. The declaration asks for it; a base rounded up at run time takes
  // the constants out of the address arithmetic (4 x 2048 tokens 574 -> 596 us, one document of 16384 4.5 % slower).
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::KV_BYTES;
  uint8_t* sQ = sV + C::KV_BYTES;                    // [STAGES]
  uint8_t* sdO = sQ + C::STAGES * C::Q_BYTES;        // [STAGES]
  uint8_t* sdST = sdO + C::STAGES * C::Q_BYTES;      // [2]
  uint8_t* sPT = sdST + 2 * C::PT_BYTES;             // [2], where it is not in TMEM
  uint8_t* sOut = sPT + (C::PT_TMEM ? 0 : 2 * C::PT_BYTES);   // [4 warpgroups][D / 32 warps]
  float* s_rows = reinterpret_cast<float*>(sOut + D / 8 * C::OUT_BYTES);  // per warpgroup: two buffers of -lse [32], -delta * scale [32]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_rows + 4 * 2 * 64);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;    // [STAGES]  (Q and dO of a stage)
  uint64_t* q_empty = bars + 4;   // [STAGES]
  uint64_t* s_full = bars + 7;    // [2]  S^T(b) and dP^T(b) ready
  uint64_t* pt_full = bars + 9;   // [2]  P^T(b) / dS^T(b) written to smem
  uint64_t* dq_full = bars + 11;  // [2]  dQ^T(b) ready (the MMAs that read P^T(b)/dS^T(b) retire before s_full of the next use)
  uint64_t* st_free = bars + 13;  // [2]  dQ^T(b) in registers: TMEM columns of b reusable
  uint64_t* acc_full = bars + 15; // dK / dV final
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&pt_full[b], 256);
      mbar_init(&dq_full[b], 1);
      mbar_init(&st_free[b], 256);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(kv_full, 2 * C::KV_BYTES);
#pragma unroll
      for (int h = 0; h < C::HALVES; ++h) {
        tma_load_2d(sK + h * HALF_BYTES, &tm_kv, kv_full, p.k_col0 + kv_head * D + h * 64, doc_start + kv0);
        tma_load_2d(sV + h * HALF_BYTES, &tm_kv, kv_full, p.v_col0 + kv_head * D + h * 64, doc_start + kv0);
      }
    }
    __syncwarp();
    int st = 0, qt = 0, head = head0;
    uint32_t ph = 0;
    for (int it = 0; it < n_iter; ++it) {
      const int qrow = doc_start + (q_first + qt) * 64 - p.q_row_off;
      if (!warp_all(mbar_wait(&q_empty[st], ph ^ 1, p.status, AXB_TIMEOUT_EMPTY))) break;
      if (elect_one()) {
        mbar_expect_tx(&q_full[st], 2 * C::Q_BYTES);
#pragma unroll
        for (int h = 0; h < C::HALVES; ++h) {
          tma_load_2d(sQ + st * C::Q_BYTES + h * C::Q_HALF, &tm_q, &q_full[st], p.q_col0 + head * D + h * 64, qrow);
          tma_load_2d(sdO + st * C::Q_BYTES + h * C::Q_HALF, &tm_do, &q_full[st], head * D + h * 64, qrow);
        }
      }
      __syncwarp();
      if (++qt == n_qt) {
        qt = 0;
        ++head;
      }
      if (++st == C::STAGES) {
        st = 0;
        ph ^= 1;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_st = make_idesc_bf16(128, 64, 0, 0);  // K/V (K-major) x Q/dO (K-major)
    constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);  // P^T/dS^T x dO/Q (MN-major)
    constexpr uint32_t idesc_dq = make_idesc_bf16(128, 64, 1, 1);  // K^T (MN) x dS^T (MN)
    constexpr uint32_t Q16 = C::Q_BYTES / 16, PT16 = C::PT_BYTES / 16;
    const uint64_t dk_k = make_smem_desc_sw128(smem_u32(sK), 16, 1024), dk_mn = make_smem_desc_sw128(smem_u32(sK), HALF_BYTES, 1024);
    const uint64_t dv_k = make_smem_desc_sw128(smem_u32(sV), 16, 1024);
    const uint64_t dq_k = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), dq_mn = make_smem_desc_sw128(smem_u32(sQ), C::Q_HALF, 1024);
    const uint64_t do_k = make_smem_desc_sw128(smem_u32(sdO), 16, 1024), do_mn = make_smem_desc_sw128(smem_u32(sdO), C::Q_HALF, 1024);
    const uint64_t ds_k = make_smem_desc_sw128(smem_u32(sdST), 16, 1024);
    const uint64_t pt_k = make_smem_desc_sw128(smem_u32(sPT), 16, 1024);
    const uint64_t ds_mn = make_smem_desc_sw128(smem_u32(sdST), HALF_BYTES, 1024);
    bool ok = warp_all(mbar_wait(kv_full, 0, p.status, AXB_TIMEOUT_FULL));
    int s_st = 0;             // stage and phase of the next scores
    uint32_t s_ph = 0;
    // S^T(i) = K . Q(i)^T and dP^T(i) = V . dO(i)^T into TMEM buffer i & 1
    auto issue_scores = [&](int i) -> bool {
      const int b = i & 1;
      bool fine = mbar_wait(&q_full[s_st], s_ph, p.status, AXB_TIMEOUT_FULL);
      // buffer b was last used by iteration i - 2: its dQ^T must have been drained
      if (fine && i >= 2) fine = mbar_wait(&st_free[b], ((i - 2) >> 1) & 1, p.status, AXB_TIMEOUT_TMEM_EMPTY);
      if (!warp_all(fine)) return false;
      tc_fence_after();
      const uint64_t dq = dq_k + (uint32_t)s_st * Q16, dd = do_k + (uint32_t)s_st * Q16;
      const uint32_t col = tmem_base + 128 * b;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {  // reduce over d
          const uint32_t koff = ((kk / 4) * HALF_BYTES + (kk % 4) * 32) / 16, qoff = ((kk / 4) * C::Q_HALF + (kk % 4) * 32) / 16;
          umma_f16(col + C::ST_COL, dk_k + koff, dq + qoff, idesc_st, kk > 0);
        }
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t koff = ((kk / 4) * HALF_BYTES + (kk % 4) * 32) / 16, qoff = ((kk / 4) * C::Q_HALF + (kk % 4) * 32) / 16;
          umma_f16(col + C::DPT_COL, dv_k + koff, dd + qoff, idesc_st, kk > 0);
        }
        umma_commit(&s_full[b]);
      }
      __syncwarp();
      if (++s_st == C::STAGES) {
        s_st = 0;
        s_ph ^= 1;
      }
      return true;
    };
    ok = ok && issue_scores(0);
    int st = 0;
    for (int it = 0; it < n_iter && ok; ++it) {
      const int b = it & 1;
      const uint32_t ph = (it >> 1) & 1;
      if (it + 1 < n_iter && !issue_scores(it + 1)) break;   // keeps the tensor core busy during softmax(it)
      const uint64_t dq = dq_mn + (uint32_t)st * Q16, dd = do_mn + (uint32_t)st * Q16;
      const uint32_t pt = tmem_base + C::DPT_COL + 128 * b;
      const uint64_t ds = ds_k + (uint32_t)b * PT16, dst = ds_mn + (uint32_t)b * PT16;
      if (!warp_all(mbar_wait(&pt_full[b], ph, p.status, AXB_TIMEOUT_GENERIC))) break;
      tc_fence_after();
      if (elect_one()) {
        // dQ^T [d, q] = K^T . dS^T over the 128 kv rows (8 K-steps of 16), into the columns of S^T(b). First, so that it is drained
        // while dV and dK run: the next scores but one wait for those columns.
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_f16(tmem_base + C::ST_COL + 128 * b, dk_mn + kk * (2048 / 16), dst + kk * (2048 / 16), idesc_dq, kk > 0);
        umma_commit(&dq_full[b]);
        // reduce over the 64 q rows of this tile: 4 K-steps of 16
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)   // dV += P^T . dO   (B = dO tile, MN-major: chunk stride = one 64x64 half)
          if (C::PT_TMEM) umma_f16_ts(tmem_base + C::DV_COL, pt + (kk >> 1) * 32 + (kk & 1) * 8, dd + kk * (2048 / 16), idesc_acc, (it > 0 || kk > 0));
          else umma_f16(tmem_base + C::DV_COL, pt_k + (uint32_t)b * PT16 + kk * 2, dd + kk * (2048 / 16), idesc_acc, (it > 0 || kk > 0));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_f16(tmem_base + C::DK_COL, ds + kk * 2, dq + kk * (2048 / 16), idesc_acc, (it > 0 || kk > 0));
        umma_commit(&q_empty[st]);
        if (it == n_iter - 1) umma_commit(acc_full);
      }
      __syncwarp();
      if (++st == C::STAGES) st = 0;
    }
  } else {
    const int lg = warp & 3;
    const int wg = (warp - 2) >> 2;    // softmax warpgroup: 32 q columns of the iterations with it % 2 == grp
    const int grp = wg >> 1, c0 = (wg & 1) * 32;
    const int r = lg * 32 + lane;      // kv row in tile (S^T, dP^T, dK, dV) or d row (dQ^T)
    const int st_tid = threadIdx.x - 64 - wg * 128;  // 0..127 inside the warpgroup
    const int kv_idx = kv0 + r;
    const uint32_t lane_off = uint32_t(lg * 32) << 16;
    const uint32_t st_addr = tmem_base + lane_off + C::ST_COL + 128 * grp + c0, dpt_addr = tmem_base + lane_off + C::DPT_COL + 128 * grp + c0;
    uint8_t* my_dst = sdST + grp * C::PT_BYTES;
    uint8_t* my_pt = sPT + grp * C::PT_BYTES;
    float* const rows = s_rows + wg * 128;
    bool ok = true;
    // -lse (so that P = exp2(S * sl2 + nlse)) or -delta * scale of one q row of iteration `it`; rows outside the document
    // or outside this rank's q window get nlse = -inf -> P = 0. Requested an iteration ahead: the trip to L2 would stand
    // in the chain from one dQ^T to the next scores otherwise.
    auto fetch_row = [&](int it) -> float {
      float val = st_tid < 32 ? -INFINITY : 0.f;
      if (it >= n_iter || st_tid >= 64) return val;
      const int q = (q_first + it % n_qt) * 64 + c0 + (st_tid & 31);
      const long long lrow = (long long)doc_start + q - p.q_row_off;
      if (q < doc_len && lrow >= 0 && lrow < p.q_rows) {
        const long long off = (long long)(head0 + it / n_qt) * p.q_rows + lrow;
        val = st_tid < 32 ? -p.lse2[off] : -p.delta[off] * p.scale;
      }
      return val;
    };
    // P^T and dS^T of 32 columns, two at a time (packed fp32 arithmetic rounds like the scalar one)
    const uint64_t sl2 = pack_f32x2(p.sl2, p.sl2), scale2 = pack_f32x2(p.scale, p.scale);
    auto gradients = [&](auto masked, const uint32_t (&sr)[32], const uint32_t (&dr)[32], const float* nlse, int qc0, int q_lo, int q_hi) {
      uint32_t pk[16];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t dk[4];
#pragma unroll
        for (int i = q * 8; i < q * 8 + 8; i += 4) {
          const ulonglong2 nl = *reinterpret_cast<const ulonglong2*>(nlse + i), ds = *reinterpret_cast<const ulonglong2*>(nlse + 32 + i);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = i + 2 * h;
            const float2 x = unpack_f32x2(fma_f32x2(pack_b32x2(sr[j], sr[j + 1]), sl2, h ? nl.y : nl.x));
            float p0 = fast_exp2(x.x), p1 = fast_exp2(x.y);
            if (decltype(masked)::value) {
              if (qc0 + j < q_lo || qc0 + j > q_hi) p0 = 0.f;
              if (qc0 + j + 1 < q_lo || qc0 + j + 1 > q_hi) p1 = 0.f;
            }
            const float2 d = unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), fma_f32x2(pack_b32x2(dr[j], dr[j + 1]), scale2, h ? ds.y : ds.x)));
            pk[j >> 1] = pack_bf16x2(p0, p1);
            dk[((i & 4) >> 1) + h] = pack_bf16x2(d.x, d.y);
          }
        }
        const uint32_t off = sw128_chunk_off(r, c0 / 8 + q);
        if (!C::PT_TMEM) *reinterpret_cast<uint4*>(my_pt + off) = make_uint4(pk[q * 4], pk[q * 4 + 1], pk[q * 4 + 2], pk[q * 4 + 3]);
        *reinterpret_cast<uint4*>(my_dst + off) = make_uint4(dk[0], dk[1], dk[2], dk[3]);
      }
      if (C::PT_TMEM) tmem_st_32x16(dpt_addr, pk);
    };
    // The sums of 32 queries (the first one `shift` rows into its group of four) leave through this warp's staging tile and bulk
    // reductions. As reductions from registers they filled the load-store queue, and the stores of the other warpgroups' dS^T stood
    // behind them: 1500 of 2800 clocks of an iteration.
    uint8_t* const out_tile = sOut + (wg * (D / 32) + lg) * C::OUT_BYTES;
    const long long width = (long long)p.Hq * D, rows4 = p.q_rows & ~3;
    auto put_rows = [&](auto shift, const uint32_t (&v)[32], int group, int col) {
      constexpr int a = decltype(shift)::value;
      constexpr bool tail = a != 0;                       // a ninth group: by itself, a 512-byte reduction
      if (lane == 0) bulk_wait_group_read<0>();           // what was staged before has left
      __syncwarp();
#pragma unroll
      for (int g = 0; g < 8 + (tail ? 1 : 0); ++g) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = 4 * g + e - a >= 0 && 4 * g + e - a < 32 ? v[(4 * g + e - a) & 31] : 0u;
        if (C::OUT_GROUPS == 4 && (g == 4 || g == 8)) {   // the tile holds four groups
          if (lane == 0) bulk_wait_group_read<0>();
          __syncwarp();
        }
        *reinterpret_cast<uint4*>(out_tile + (C::OUT_GROUPS == 4 ? g & 3 : g) * 512 + lane * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        if ((C::OUT_GROUPS == 4 && g == 3) || g == 7 || g == 8) {
          if (g == 7 && tail && C::OUT_GROUPS == 8) continue;   // both leave after the ninth
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (g < 8) tma_reduce_add_2d(&tm_dq, out_tile, col, group + (g & ~(C::OUT_GROUPS - 1)));
            else {
              if (C::OUT_GROUPS == 8) tma_reduce_add_2d(&tm_dq, out_tile, col, group);
              bulk_reduce_add_f32(p.dq_acc + (group + 8) * 4 * width + col, out_tile + (C::OUT_GROUPS == 4 ? 0 : 8) * 512, 512);
            }
            bulk_commit_group();
          }
        }
      }
    };
    float row_val = fetch_row(grp);
    if (st_tid < 64) rows[st_tid] = row_val;
    row_val = fetch_row(grp + 2);
    asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");
    for (int it = grp; it < n_iter; it += 2) {
      const uint32_t ph = (it >> 1) & 1;
      const int head = head0 + it / n_qt;
      const int qt0 = (q_first + it % n_qt) * 64;  // doc-relative first q row of the tile
      const int qc0 = qt0 + c0;                    // ... and of this group's columns
      const float* nlse = rows + ph * 64;
      // (a lane whose wait ran out walks on with the others, without waiting again: the group meets at the barrier below)
      ok = ok && mbar_wait(&s_full[grp], ph, p.status, AXB_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      // Only tiles that touch the diagonal or the end of the document need per-element masks
      // (q rows outside the document already carry nlse = -inf, i.e. P = 0).
      const bool need_mask = (!bidir && qc0 < kv0 + 127) || (kv0 + 128 > doc_len) || (win > 0 && qc0 + 31 >= kv0 + win);
      {
        uint32_t sr[32], dr[32];
        tmem_ld_32x32(st_addr, sr);
        tmem_ld_32x32(dpt_addr, dr);
        tmem_ld_wait();
        if (need_mask) {
          const bool row_in_doc = kv_idx < doc_len;
          // q rows that see this thread's kv row: [q_lo, q_hi] (empty for kv rows beyond the document)
          const int q_lo = row_in_doc ? (bidir ? -(1 << 30) : kv_idx) : (1 << 30);
          const int q_hi = win > 0 ? kv_idx + win - 1 : (1 << 30);
          gradients(std::true_type{}, sr, dr, nlse, qc0, q_lo, q_hi);
        } else {
          gradients(std::false_type{}, sr, dr, nlse, 0, 0, 0);
        }
      }
      if (C::PT_TMEM) tmem_st_wait();
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(&pt_full[grp]);
      // lse / delta of this group's next iteration into the other buffer, while the MMAs run; the barrier also says that all warps of
      // the group have read the present one
      if (st_tid < 64) rows[(ph ^ 1) * 64 + st_tid] = row_val;
      row_val = fetch_row(it + 4);
      asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");
      // drain dQ^T: this thread owns d = r (only rows < D are meaningful)
      ok = ok && mbar_wait(&dq_full[grp], ph, p.status, AXB_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      {
        // valid q columns of this group: inside the document and inside this rank's q window
        const long long row0 = (long long)doc_start + qc0 - p.q_row_off;   // local row of column 0
        int i_lo = row0 < 0 ? (int)(-row0) : 0;
        int i_hi = min(32, doc_len - qc0);
        if (row0 + i_hi > p.q_rows) i_hi = (int)(p.q_rows - row0);
        uint32_t qr[32];
        tmem_ld_32x32(st_addr, qr);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(&st_free[grp]);      // the next scores may overwrite the columns while the sums leave
        if (r < D) {
          if (row0 >= 0 && ((row0 + 31) | 3) < rows4) {      // every group that these rows touch is one of four whole rows
            if (i_hi < 32) {
#pragma unroll
              for (int i = 0; i < 32; ++i) qr[i] = i < i_hi ? qr[i] : 0u;
            }
            const int group = (int)(row0 >> 2), col = head * (4 * D) + lg * 128;
            switch ((int)(row0 & 3)) {
              case 0: put_rows(std::integral_constant<int, 0>{}, qr, group, col); break;
              case 1: put_rows(std::integral_constant<int, 1>{}, qr, group, col); break;
              case 2: put_rows(std::integral_constant<int, 2>{}, qr, group, col); break;
              default: put_rows(std::integral_constant<int, 3>{}, qr, group, col); break;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i >= i_lo && i < i_hi) atomicAdd(p.dq_acc + dq_at(row0 + i, (long long)head * D + r, width, rows4), __uint_as_float(qr[i]));
          }
        }
      }
    }
    if (lane == 0) bulk_wait_group<0>();
    // final dK / dV: 32 columns of each per warpgroup
    if (warp_all(ok && wg < D / 32 && mbar_wait(acc_full, 0, p.status, AXB_TIMEOUT_TMEM_FULL))) {
      tc_fence_after();
      const bool row_ok = kv_idx < doc_len && n_iter > 0;
      const long long grow = (long long)doc_start + kv_idx;  // global kv row
      __nv_bfloat16* base = p.dkv;
      long long brow = grow;
      if (p.cp_world > 1) {
        const long long owner = min(grow / p.cp_chunk, (long long)p.cp_world - 1);
        base = reinterpret_cast<__nv_bfloat16*>(p.cp_dkv_ptrs[owner]);
        brow = grow - owner * p.cp_chunk;
      }
      __nv_bfloat16* krow = base + brow * p.dkv_ld + p.dk_col0 + (long long)kv_head * D;
      __nv_bfloat16* vrow = base + brow * p.dkv_ld + p.dv_col0 + (long long)kv_head * D;
      {
        const int c = wg;
        uint32_t a[32], b[32];
        tmem_ld_32x32(tmem_base + lane_off + C::DK_COL + c * 32, a);
        tmem_ld_32x32(tmem_base + lane_off + C::DV_COL + c * 32, b);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 u, w;
            u.x = pack_bf16x2(__uint_as_float(a[q * 8 + 0]), __uint_as_float(a[q * 8 + 1]));
            u.y = pack_bf16x2(__uint_as_float(a[q * 8 + 2]), __uint_as_float(a[q * 8 + 3]));
            u.z = pack_bf16x2(__uint_as_float(a[q * 8 + 4]), __uint_as_float(a[q * 8 + 5]));
            u.w = pack_bf16x2(__uint_as_float(a[q * 8 + 6]), __uint_as_float(a[q * 8 + 7]));
            w.x = pack_bf16x2(__uint_as_float(b[q * 8 + 0]), __uint_as_float(b[q * 8 + 1]));
            w.y = pack_bf16x2(__uint_as_float(b[q * 8 + 2]), __uint_as_float(b[q * 8 + 3]));
            w.z = pack_bf16x2(__uint_as_float(b[q * 8 + 4]), __uint_as_float(b[q * 8 + 5]));
            w.w = pack_bf16x2(__uint_as_float(b[q * 8 + 6]), __uint_as_float(b[q * 8 + 7]));
            if (p.cp_world > 1 || p.kv_split > 1) {
              asm volatile("red.relaxed.sys.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(
                               krow + c * 32 + q * 8),
                           "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w)
                           : "memory");
              asm volatile("red.relaxed.sys.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(
                               vrow + c * 32 + q * 8),
                           "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w)
                           : "memory");
            } else {
              *reinterpret_cast<uint4*>(krow + c * 32 + q * 8) = u;
              *reinterpret_cast<uint4*>(vrow + c * 32 + q * 8) = w;
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

template <int D>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tm, const AttnParams& p, cudaStream_t st) {
  using C = FwdCfg<D>;
  auto kern = flash_fwd_kernel<D>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  dim3 grid(p.pair_mode == 1 ? p.Hq / 2 : p.Hq, p.n_tiles);
  kern<<<grid, kFwdThreads, C::SMEM, st>>>(tq, tm, p);
  return (int)cudaGetLastError();
}
template <int D>
int launch_bwd(const CUtensorMap& tkv, const CUtensorMap& tq, const CUtensorMap& tdo,
               const AttnParams& p, cudaStream_t st) {
  using C = BwdCfg<D>;
  CUtensorMap tdq;     // without a whole group of four rows nothing goes through it
  if (axb_make_tmap_2d(&tdq, p.dq_acc, p.T >= 4 ? p.T / 4 : 1, 4ll * p.Hq * D, 4ll * p.Hq * D, C::OUT_GROUPS, 128, 4, false)) return -4;
  auto kern = flash_bwd_kernel<D>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  dim3 grid(p.Hk * p.kv_split, p.n_tiles);
  kern<<<grid, kBwdThreads, C::SMEM, st>>>(tkv, tq, tdo, tdq, p);
  return (int)cudaGetLastError();
}
}  // namespace

namespace {

struct AttnGeom {
  const void* q_buf;   // rows [q_row_off, q_row_off + q_rows) of the token stream; q heads at q_col0
  long long q_ld;
  long long q_rows;
  int q_row_off;
  const void* kv_buf;  // all kv_rows rows; k heads at k_col0, v heads at v_col0
  long long kv_ld;
  long long kv_rows;
};

int flash_fwd_impl(const AttnGeom& g, int Hq, int Hk, int D, int q_col0, int k_col0, int v_col0,
                   const void* tiles, int n_tiles, void* out, long long out_ld, float* lse2,
                   float softmax_scale, int* status, void* stream) {
  if (g.q_rows <= 0 || n_tiles <= 0) return 0;
  if (D != 64 && D != 128) return -2;
  if ((g.q_ld & 7) || (g.kv_ld & 7) || (out_ld & 7) || (q_col0 & 7) || (k_col0 & 7) || (v_col0 & 7)) return -3;
  CUtensorMap tq, tkv;
  if (axb_make_tmap_2d(&tq, g.q_buf, g.q_rows, g.q_ld, g.q_ld, 128, 64)) return -4;
  if (axb_make_tmap_2d(&tkv, g.kv_buf, g.kv_rows, g.kv_ld, g.kv_ld, 128, 64)) return -4;
  AttnParams p = {};
  p.tiles = reinterpret_cast<const int4*>(tiles);
  p.n_tiles = n_tiles;
  p.Hq = Hq;
  p.Hk = Hk;
  p.q_col0 = q_col0;
  p.k_col0 = k_col0;
  p.v_col0 = v_col0;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.out_ld = out_ld;
  p.lse2 = lse2;
  p.T = g.q_rows;
  p.kv_rows = g.kv_rows;
  p.q_row_off = g.q_row_off;
  p.q_rows = (int)g.q_rows;
  p.sl2 = softmax_scale * 1.4426950408889634f;
  p.scale = softmax_scale;
  p.status = status;
  // Two heads share K / V and have the same blocks, so they pair wherever the group is even. Odd groups pair neighbouring q
  // tiles; a table that holds only the tiles of a rank's rows may lack one of the two, so those run single units.
  p.pair_mode = (Hq / Hk) % 2 == 0 ? 1 : (g.q_rows == g.kv_rows && g.q_row_off == 0 ? 2 : 0);
  // A pair takes about 1.25 times a single unit's time, so with fewer pairs than three quarters of the SMs single units
  // finish first (6 heads, 500 + 300 tokens: 18 us single, 23 us paired; 8 heads, 2 x 2048: 44 / 47 us). From there to two
  // units an SM it depends on the lengths, which the table's owner knows and this function does not (222 to 296 units: 0.80
  // to 1.32 times as fast in pairs, level on average); above, pairs are 1.1 to 1.5 times as fast.
  if (2ll * 111 > (long long)Hq * n_tiles) p.pair_mode = 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return D == 128 ? launch_fwd<128>(tq, tkv, p, st) : launch_fwd<64>(tq, tkv, p, st);
}

int flash_bwd_impl(const AttnGeom& g, const void* dout, const void* out, long long o_ld, const float* lse2,
                   int Hq, int Hk, int D, int q_col0, int k_col0, int v_col0, const void* tiles, int n_tiles,
                   void* dqkv, long long dqkv_ld, int dq_col0, int dk_col0, int dv_col0, float* dq_acc,
                   float* delta, float softmax_scale, int cp_world, long long cp_chunk,
                   const unsigned long long* cp_dkv_ptrs, int* status, void* stream) {
  if (g.q_rows <= 0 || n_tiles <= 0) return 0;
  if (D != 64 && D != 128) return -2;
  if ((g.q_ld & 7) || (g.kv_ld & 7) || (o_ld & 7) || (dqkv_ld & 7) || cp_world > 8) return -3;
  if (!attn_bwd_aligned(out, dqkv, dq_acc)) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long long T = g.q_rows;
  CUtensorMap tkv, tq, tdo;
  if (axb_make_tmap_2d(&tkv, g.kv_buf, g.kv_rows, g.kv_ld, g.kv_ld, 128, 64)) return -4;
  if (axb_make_tmap_2d(&tq, g.q_buf, T, g.q_ld, g.q_ld, 64, 64)) return -4;
  if (axb_make_tmap_2d(&tdo, dout, T, (long long)Hq * D, o_ld, 64, 64)) return -4;
  cudaError_t e = cudaMemsetAsync(dq_acc, 0, sizeof(float) * T * Hq * D, st);
  if (e != cudaSuccess) return (int)e;
  if (D == 128) launch_attn_delta<128>(dout, out, delta, T, Hq, o_ld, st);
  else launch_attn_delta<64>(dout, out, delta, T, Hq, o_ld, st);
  AttnParams p = {};
  p.tiles = reinterpret_cast<const int4*>(tiles);
  p.n_tiles = n_tiles;
  p.Hq = Hq;
  p.Hk = Hk;
  p.q_col0 = q_col0;
  p.k_col0 = k_col0;
  p.v_col0 = v_col0;
  p.lse2 = const_cast<float*>(lse2);
  p.T = T;
  p.kv_rows = g.kv_rows;
  p.q_row_off = g.q_row_off;
  p.q_rows = (int)T;
  p.sl2 = softmax_scale * 1.4426950408889634f;
  p.scale = softmax_scale;
  p.status = status;
  p.delta = delta;
  p.dq_acc = dq_acc;
  p.dkv = reinterpret_cast<__nv_bfloat16*>(dqkv);
  p.dkv_ld = dqkv_ld;
  p.dk_col0 = dk_col0;
  p.dv_col0 = dv_col0;
  p.cp_world = cp_world > 1 ? cp_world : 1;
  p.cp_chunk = cp_chunk;
  // Wide GQA groups: one CTA per (kv tile, kv head) loops over group * q-tiles iterations, and the
  // longest such CTA bounds the launch. Two CTAs per kv head halve it; their dK / dV partials meet
  // in the (zeroed) gradient buffer through bf16x2 reduce-adds.
  p.kv_split = (cp_world <= 1 && Hq / Hk >= 8 && (Hq / Hk) % 2 == 0 && dv_col0 == dk_col0 + Hk * D) ? 2 : 1;
  if (p.kv_split > 1) {
    e = cudaMemset2DAsync(reinterpret_cast<__nv_bfloat16*>(dqkv) + dk_col0, (size_t)dqkv_ld * 2, 0,
                          (size_t)2 * Hk * D * 2, (size_t)g.kv_rows, st);
    if (e != cudaSuccess) return (int)e;
  }
  for (int i = 0; i < 8; ++i) p.cp_dkv_ptrs[i] = (cp_world > 1 && i < cp_world) ? cp_dkv_ptrs[i] : 0ull;
  int rc = D == 128 ? launch_bwd<128>(tkv, tq, tdo, p, st) : launch_bwd<64>(tkv, tq, tdo, p, st);
  if (rc) return rc;
  launch_dq_convert(dq_acc, dqkv, T, Hq * D, dqkv_ld, dq_col0, st);
  return (int)cudaGetLastError();
}

}  // namespace

// qkv: fused projection [T, ld] bf16 with q heads at column q_col0, k heads at k_col0, v at
// v_col0 (head-major, D per head). tiles: device int4 array built by axb_build_attn_tiles
// (tile rows = 128). out: [T, out_ld] bf16, lse2: [Hq, T] fp32.
extern "C" int axb_flash_varlen_fwd(const void* qkv, long long ld, long long T, int Hq, int Hk,
                                    int D, int q_col0, int k_col0, int v_col0, const void* tiles,
                                    int n_tiles, void* out, long long out_ld, float* lse2,
                                    float softmax_scale, int* status, void* stream) {
  AttnGeom g = {qkv, ld, T, 0, qkv, ld, T};
  return flash_fwd_impl(g, Hq, Hk, D, q_col0, k_col0, v_col0, tiles, n_tiles, out, out_ld, lse2,
                        softmax_scale, status, stream);
}

// Backward. dout/out: [T, o_ld] bf16; dqkv: fused gradient buffer with the layout of qkv (all
// three blocks are written); dq_acc: T * Hq * D fp32 of scratch (zeroed here; 16-byte aligned); delta: fp32 [Hq, T]
// scratch. tiles must have been built with 128-row tiles.
extern "C" int axb_flash_varlen_bwd(const void* qkv, long long ld, const void* dout,
                                    const void* out, long long o_ld, const float* lse2,
                                    long long T, int Hq, int Hk, int D, int q_col0, int k_col0,
                                    int v_col0, const void* tiles, int n_tiles, void* dqkv,
                                    long long dqkv_ld, float* dq_acc, float* delta,
                                    float softmax_scale, int* status, void* stream) {
  AttnGeom g = {qkv, ld, T, 0, qkv, ld, T};
  return flash_bwd_impl(g, dout, out, o_ld, lse2, Hq, Hk, D, q_col0, k_col0, v_col0, tiles, n_tiles, dqkv,
                        dqkv_ld, q_col0, k_col0, v_col0, dq_acc, delta, softmax_scale, 1, 0, nullptr, status,
                        stream);
}

// Context-parallel forward: q rows [q_row_off, q_row_off + q_rows) come from the local fused
// projection `q_buf`; K and V of the WHOLE token stream come from `kv_buf` ([kv_rows, kv_ld], k
// heads at column 0, v heads at Hk*D), which the ranks filled by storing their rows into every
// peer's buffer. tiles: (doc_start, doc_len, tile_start) in GLOBAL rows, only tiles that
// intersect the local q rows. out [q_rows, out_ld], lse2 [Hq, q_rows].
extern "C" int axb_flash_varlen_fwd_cp(const void* q_buf, long long q_ld, long long q_rows, int q_row_off,
                                       const void* kv_buf, long long kv_ld, long long kv_rows, int Hq,
                                       int Hk, int D, const void* tiles, int n_tiles, void* out,
                                       long long out_ld, float* lse2, float softmax_scale, int* status,
                                       void* stream) {
  AttnGeom g = {q_buf, q_ld, q_rows, q_row_off, kv_buf, kv_ld, kv_rows};
  return flash_fwd_impl(g, Hq, Hk, D, 0, 0, Hk * D, tiles, n_tiles, out, out_ld, lse2, softmax_scale, status,
                        stream);
}

// Context-parallel backward: dQ of the local rows goes to the q block of `dqkv` ([q_rows, dqkv_ld],
// fused layout); the dK / dV tiles this rank computes for ANY kv row are reduce-added over NVLink
// into the k / v blocks of the owner's gradient buffer cp_dkv_ptrs[row / cp_chunk] (HOST array of
// peer-mapped addresses, same fused layout, zeroed by the caller before any rank starts).
extern "C" int axb_flash_varlen_bwd_cp(const void* q_buf, long long q_ld, long long q_rows, int q_row_off,
                                       const void* kv_buf, long long kv_ld, long long kv_rows,
                                       const void* dout, const void* out, long long o_ld, const float* lse2,
                                       int Hq, int Hk, int D, const void* tiles, int n_tiles, void* dqkv,
                                       long long dqkv_ld, float* dq_acc, float* delta, float softmax_scale,
                                       int cp_world, long long cp_chunk,
                                       const unsigned long long* cp_dkv_ptrs, int* status, void* stream) {
  AttnGeom g = {q_buf, q_ld, q_rows, q_row_off, kv_buf, kv_ld, kv_rows};
  return flash_bwd_impl(g, dout, out, o_ld, lse2, Hq, Hk, D, 0, 0, Hk * D, tiles, n_tiles, dqkv, dqkv_ld, 0,
                        Hq * D, (Hq + Hk) * D, dq_acc, delta, softmax_scale, cp_world, cp_chunk, cp_dkv_ptrs,
                        status, stream);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of the backward pass (declared and documented in axb_noalloc.h): the
// dQ accumulator and the delta vector live in a fixed device array inside this library instead
// of caller-provided scratch, for callers that cannot allocate device memory.
#include <cstdio>

#include "axb_noalloc.h"

static __device__ __align__(256) float
    g_noalloc_scratch[AXB_NOALLOC_MAX_DQ_FLOATS + AXB_NOALLOC_MAX_DELTA_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
float* g_noalloc_ptr[kMaxDevices] = {nullptr};

void set_err(char* err, int err_len, const char* msg) {
  if (err && err_len > 0) std::snprintf(err, (size_t)err_len, "%s", msg);
}
}  // namespace

extern "C" int axb_flash_varlen_bwd_noalloc(const void* qkv, long long ld, const void* dout,
                                            const void* out, long long o_ld, const float* lse2,
                                            long long T, int Hq, int Hk, int D, int q_col0,
                                            int k_col0, int v_col0, const void* tiles, int n_tiles,
                                            void* dqkv, long long dqkv_ld, float softmax_scale,
                                            int* status, void* stream, char* err, int err_len) {
  if (T < 0 || Hq <= 0 || D <= 0) {
    set_err(err, err_len, "axb_flash_varlen_bwd_noalloc: T must be >= 0 and Hq, D must be positive");
    return AXB_NOALLOC_BAD_SIZE;
  }
  if (T == 0 || n_tiles <= 0) return 0;  // an empty batch: nothing to compute, nothing launched
  const long long dq_floats = T * (long long)Hq * D;
  const long long delta_floats = T * (long long)Hq;
  if (dq_floats > AXB_NOALLOC_MAX_DQ_FLOATS || delta_floats > AXB_NOALLOC_MAX_DELTA_FLOATS) {
    char msg[256];
    std::snprintf(msg, sizeof(msg),
                  "axb_flash_varlen_bwd_noalloc: T*Hq*D = %lld (max %d) or T*Hq = %lld (max %d) "
                  "exceeds the built-in scratch array; use axb_flash_varlen_bwd with your own scratch",
                  dq_floats, AXB_NOALLOC_MAX_DQ_FLOATS, delta_floats, AXB_NOALLOC_MAX_DELTA_FLOATS);
    set_err(err, err_len, msg);
    return AXB_NOALLOC_TOO_LARGE;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    set_err(err, err_len, "axb_flash_varlen_bwd_noalloc: no current CUDA device");
    return AXB_NOALLOC_SETUP_FAILED;
  }
  if (g_noalloc_ptr[dev] == nullptr) {
    // one-time set-up per device: in host code the array's name is only a stand-in, the kernels
    // need its device address
    float* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_err(err, err_len, cudaGetErrorString(e));
      return AXB_NOALLOC_SETUP_FAILED;
    }
    g_noalloc_ptr[dev] = p;
  }
  float* dq_acc = g_noalloc_ptr[dev];
  float* delta = g_noalloc_ptr[dev] + AXB_NOALLOC_MAX_DQ_FLOATS;
  // the callee clears dq_acc (it must start at zero) and overwrites delta completely
  const int rc = axb_flash_varlen_bwd(qkv, ld, dout, out, o_ld, lse2, T, Hq, Hk, D, q_col0, k_col0,
                                      v_col0, tiles, n_tiles, dqkv, dqkv_ld, dq_acc, delta,
                                      softmax_scale, status, stream);
  if (rc != 0) set_err(err, err_len, "axb_flash_varlen_bwd_noalloc: kernel launch failed");
  return rc;
}
