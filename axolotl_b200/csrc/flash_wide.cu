// Packed variable-length flash attention for WIDE heads on sm_100a: q/k head width 192 or 256, v head width
// 128 or 256 (Gemma 1/2/3 with head_dim 256; multi-head latent attention with 192-wide q/k and 128-wide v),
// optional tanh soft-capping of the scores (Gemma 2), causal or bidirectional documents, sliding windows.
//
// The 128-wide kernels of flash_varlen.cu keep a whole head in shared memory and TMEM with double buffers;
// at 256 that does not fit (Q + K + V tiles of 128 rows are 192 KB, dK + dV accumulators are all 512 TMEM
// columns).
//   forward   grid (q head, q tile): Q stays, K and V stream through a ring of 128-column units
//   backward  grid (kv head, kv tile, part): S^T, dP^T over the full widths; dV[:, part], dK[:, part] and
//             dQ^T[part, :] of one 128-column PART of the outputs, so the score GEMMs are computed once per part
//             (1.4x the minimum FLOPs at 256/256) and nothing else grows. Stages are single-buffered.
// Same tile table, same packed fused-projection layout [T, Hq*Dqk | Hk*Dqk | Hk*Dv] and the same bounded waits as
// flash_varlen.cu.
//
// Takes the place of the reference's flash-attn / SDPA paths for these head sizes
// (src/axolotl/monkeypatch/attention/flash_attn_4.py:37-111; Gemma attention soft-capping reaches the
// reference through HF's eager/flash paths selected in src/axolotl/loaders/model.py:560-640).
#include "attn_common.cuh"
#include <type_traits>

namespace {

constexpr int HALF_BYTES = 128 * 128;  // 128 rows x 128 B (64 bf16), swizzled
constexpr int QH_BYTES = 64 * 128;     // 64 rows x 128 B

struct WideParams {
  const int4* tiles;  // (doc_start, doc_len, tile_start, flags: bit 0 bidirectional, bits 1.. sliding window)
  int n_tiles;
  int Hq, Hk;
  int q_col0, k_col0, v_col0;
  __nv_bfloat16* out;  // [T, Hq * Dv]
  long long out_ld;
  float* lse2;         // [Hq, T], log2 domain
  long long T;
  float sl2;           // softmax_scale * log2(e)
  float scale;
  float cap_in;        // soft cap: u = s * cap_in (= scale / cap); effective score (log2 domain) = tanh(u) * cap_out2
  float cap_out2;      // cap * log2(e)
  int* status;
  // backward
  const float* delta;  // [Hq, T]
  float* dq_acc;       // T * Hq * Dqk fp32 in the order of dq_at, accumulated with reductions
  __nv_bfloat16* dkv;  // gradient buffer, same layout as qkv
  long long dkv_ld;
  int dk_col0, dv_col0;
};

// =====================================================================================================
// Forward: 192 threads = TMA warp, MMA warp, 4 softmax warps. One CTA per (q head, 128-row q tile), all of the v head.
// S is double buffered in TMEM [S0 | S1 | O (Dv)]: the scores of the next block are there when a block's P is done, and the next
// but one are issued behind its P.V. P (bf16) overwrites the first half of its S columns and is the TMEM operand of P.V. O
// accumulates in TMEM and is rescaled by a warp that has a row with a new maximum (see flash_varlen.cu).
// K and V stream through one ring of 128-column units in the order in which the MMA warp reads them: K(0), K(1), V(0), K(2),
// V(1), ... Q and the ring's five units fill shared memory.
// Bound: the load latency of a unit against the ring, then the MMA stream (2048 clocks per 128 x 128 block at 256 / 256).
// 4 documents of 2048, 16 / 8 heads of 256: 363 -> 166 us against one CTA per 128-column part of V with S, softmax and P (through
// shared memory) done once per part, O in registers and single K / V buffers.
// =====================================================================================================
template <int DQK, int DV>
struct WFwd {
  static constexpr int QK_BYTES = (DQK / 64) * HALF_BYTES;
  static constexpr int KU = (DQK + 127) / 128, VU = DV / 128;   // units of a K / V tile (the last of a 192-wide K is half full)
  static constexpr int UNIT = 2 * HALF_BYTES, SLOTS = 5;
  static constexpr int SMEM = QK_BYTES + SLOTS * UNIT + 1024 + 256;
  static constexpr int O_COL = 256;
  static_assert(SMEM <= 227 * 1024 && O_COL + DV <= 512, "");
};

template <int DQK, int DV, bool SOFTCAP>
__global__ void __launch_bounds__(192, 1)
    flash_wide_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv,
                          const WideParams p) {
  using C = WFwd<DQK, DV>;
  const int tile_id = blockIdx.y;
  if (tile_id >= p.n_tiles) return;
  const int head = blockIdx.x;
  const int kv_head = head / (p.Hq / p.Hk);
  const int4 ti = p.tiles[tile_id];
  const int doc_start = ti.x, doc_len = ti.y, q0 = ti.z;
  if (!AXB_INDEX_OK(AXB_SITE_ATTN_TILE, (long long)doc_start + doc_len - 1, p.T) || !AXB_INDEX_OK(AXB_SITE_ATTN_TILE, q0, doc_len)) return;
  const bool bidir = ti.w & 1;
  const int win = bidir ? 0 : (ti.w >> 1);
  const int kv_end = bidir ? doc_len : min(q0 + 128, doc_len);
  const int jb0 = win > 0 ? max(0, q0 - win + 1) / 128 : 0;
  const int n_blocks = (kv_end + 127) / 128 - jb0;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sU = sQ + C::QK_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sU + C::SLOTS * C::UNIT);
  uint64_t* q_full = bars + 0;
  uint64_t* u_full = bars + 1;               // [slot] unit landed
  uint64_t* u_empty = u_full + C::SLOTS;     // [slot] its MMAs retired
  uint64_t* s_full = u_empty + C::SLOTS;     // [2] scores ready
  uint64_t* p_full = s_full + 2;             // [2] P written (S read, O rescaled)
  uint64_t* pv_full = p_full + 2;            // [2] P.V added to O
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_full + 2);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < C::SLOTS; ++s) {
      mbar_init(&u_full[s], 1);
      mbar_init(&u_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 128);
      mbar_init(&pv_full[s], 1);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tm_kv);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 2) {
    int slot = 0;                            // both warps walk the units in the same order
    uint32_t phase = 0;
    auto advance = [&]() {
      if (++slot == C::SLOTS) {
        slot = 0;
        phase ^= 1;
      }
    };
    if (warp == 0) {
      if (elect_one()) {
        mbar_expect_tx(q_full, C::QK_BYTES);
#pragma unroll
        for (int h = 0; h < DQK / 64; ++h)
          tma_load_2d(sQ + h * HALF_BYTES, &tm_q, q_full, p.q_col0 + head * DQK + h * 64, doc_start + q0);
      }
      __syncwarp();
      // columns col0 .. col0 + width - 1 of block j, in units
      auto load = [&](int j, int col0, int width) -> bool {
        for (int c = 0; c < width; c += 128, advance()) {
          if (!warp_all(mbar_wait(&u_empty[slot], phase ^ 1, p.status, AXB_TIMEOUT_EMPTY))) return false;
          const int halves = width - c >= 128 ? 2 : 1;
          if (elect_one()) {
            mbar_expect_tx(&u_full[slot], halves * HALF_BYTES);
            for (int h = 0; h < halves; ++h)
              tma_load_2d(sU + slot * C::UNIT + h * HALF_BYTES, &tm_kv, &u_full[slot], col0 + c + h * 64, doc_start + (jb0 + j) * 128);
          }
          __syncwarp();
        }
        return true;
      };
      const int kc = p.k_col0 + kv_head * DQK, vc = p.v_col0 + kv_head * DV;
      bool ok = true;
      for (int j = 0; j < 2 && j < n_blocks && ok; ++j) ok = load(j, kc, DQK);
      for (int j = 0; j < n_blocks && ok; ++j) {
        ok = load(j, vc, DV);
        if (ok && j + 2 < n_blocks) ok = load(j + 2, kc, DQK);
      }
    } else {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc_bf16(128, 128, 0, 1);
      const uint64_t dq = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), dk_base = make_smem_desc_sw128(smem_u32(sU), 16, 1024);
      const uint64_t dv_base = make_smem_desc_sw128(smem_u32(sU), HALF_BYTES, 1024);
      auto issue_s = [&](int j) -> bool {
        const int b = j & 1;
#pragma unroll
        for (int u = 0; u < C::KU; ++u, advance()) {
          if (!warp_all(mbar_wait(&u_full[slot], phase, p.status, AXB_TIMEOUT_FULL))) return false;
          tc_fence_after();
          const uint64_t dk = dk_base + (uint32_t)(slot * (C::UNIT / 16));
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              if (u * 128 + kk * 16 >= DQK) break;
              const uint32_t off = ((kk / 4) * HALF_BYTES + (kk % 4) * 32) / 16;
              umma_f16(tmem_base + b * 128, dq + u * (C::UNIT / 16) + off, dk + off, idesc_s, u > 0 || kk > 0);
            }
            umma_commit(&u_empty[slot]);
            if (u == C::KU - 1) umma_commit(&s_full[b]);
          }
          __syncwarp();
        }
        return true;
      };
      auto issue_pv = [&](int j) -> bool {
        const int b = j & 1;
        if (!warp_all(mbar_wait(&p_full[b], (j >> 1) & 1, p.status, AXB_TIMEOUT_GENERIC))) return false;
#pragma unroll
        for (int u = 0; u < C::VU; ++u, advance()) {
          if (!warp_all(mbar_wait(&u_full[slot], phase, p.status, AXB_TIMEOUT_FULL))) return false;
          tc_fence_after();
          const uint64_t dv = dv_base + (uint32_t)(slot * (C::UNIT / 16));
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)       // 128 kv rows / 16: 8 TMEM columns of P each
              umma_f16_ts(tmem_base + C::O_COL + u * 128, tmem_base + b * 128 + kk * 8, dv + kk * (2048 / 16), idesc_pv, j > 0 || kk > 0);
            umma_commit(&u_empty[slot]);
            if (u == C::VU - 1) umma_commit(&pv_full[b]);
          }
          __syncwarp();
        }
        return true;
      };
      bool ok = n_blocks > 0 && warp_all(mbar_wait(q_full, 0, p.status, AXB_TIMEOUT_FULL));
      for (int j = 0; j < 2 && j < n_blocks && ok; ++j) ok = issue_s(j);
      for (int j = 0; j < n_blocks && ok; ++j) {
        ok = issue_pv(j);
        if (ok && j + 2 < n_blocks) ok = issue_s(j + 2);     // over P(j), which the P.V before it has read
      }
    }
  } else {
    const int lg = warp & 3;
    const int r = lg * 32 + lane;
    const int q_idx = q0 + r;
    const uint32_t lane_off = uint32_t(lg * 32) << 16;
    const uint32_t o_addr = tmem_base + lane_off + C::O_COL;
    const float mul = SOFTCAP ? 1.f : p.sl2;      // to the log2 domain (soft-capped scores are brought there first)
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_blocks && ok; ++j) {
      const int b = j & 1;
      if (!warp_all(mbar_wait(&s_full[b], (j >> 1) & 1, p.status, AXB_TIMEOUT_TMEM_FULL))) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t s_addr = tmem_base + lane_off + b * 128;
      uint32_t sr[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, sr[c]);
      tmem_ld_wait();
      if constexpr (SOFTCAP) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) sr[c][i] = __float_as_uint(tanhf(__uint_as_float(sr[c][i]) * p.cap_in) * p.cap_out2);
      }
      const int kv0 = (jb0 + j) * 128;
      if (kv0 + 127 > (bidir ? doc_len - 1 : min(q0, doc_len - 1)) || (win > 0 && kv0 < q0 + 128 - win)) {
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
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * mul);
      if (j == 0) {
        m = m_new;
      } else if (__any_sync(0xffffffffu, m_new > m)) {
        // S(j) was issued behind P.V(j - 2): the one after it has to be waited for
        if (!warp_all(mbar_wait(&pv_full[b ^ 1], ((j - 1) >> 1) & 1, p.status, AXB_TIMEOUT_TMEM_FULL))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const float alpha = m_new == m ? 1.f : fast_exp2(m - m_new);
        m = m_new;
        l *= alpha;
#pragma unroll 1
        for (int c = 0; c < DV / 64; ++c) {
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
          const float p0 = fast_exp2(fmaf(__uint_as_float(sr[c][i]), mul, -m_use));
          const float p1 = fast_exp2(fmaf(__uint_as_float(sr[c][i + 1]), mul, -m_use));
          sum[i & 2] += p0;
          sum[(i & 2) + 1] += p1;
          pk[i >> 1] = pack_bf16x2(p0, p1);
        }
        tmem_st_32x16(s_addr + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[b]);
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
    const int last = n_blocks - 1;
    if (ok && n_blocks > 0 && warp_all(mbar_wait(&pv_full[last & 1], (last >> 1) & 1, p.status, AXB_TIMEOUT_TMEM_FULL))) {
      tc_fence_after();
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      const long long row = (long long)doc_start + q_idx;
      const bool row_ok = q_idx < doc_len && row < p.T;
      __nv_bfloat16* orow = p.out + row * p.out_ld + (long long)head * DV;
#pragma unroll 1
      for (int c = 0; c < DV / 32; ++c) {
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
      if (row_ok) p.lse2[(long long)head * p.T + row] = m + log2f(l);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// =====================================================================================================
// Backward: 576 threads = TMA warp, MMA warp, four softmax warpgroups. One CTA per (kv head, 128-row kv tile,
// part); loops over the q heads of the GQA group and the 64-row q tiles that see the kv tile. Per iteration
//   S^T [kv, q] = K . Q^T (over Dqk)      dP^T [kv, q] = V . dO^T (over Dv)
//   dV[:, part] += P^T . dO[:, part]      dK[:, part] += dS^T . Q[:, part]
//   dQ^T[part, q] = K[:, part]^T . dS^T   (fp32 reductions into dq_acc)
// A 192-wide q/k head has the parts [0, 128) and [64, 192): the second stores only its upper 64 columns.
// =====================================================================================================
template <int DQK, int DV>
struct WBwd {
  static constexpr int K_BYTES = (DQK / 64) * HALF_BYTES;
  static constexpr int V_BYTES = (DV / 64) * HALF_BYTES;
  static constexpr int Q_BYTES = (DQK / 64) * QH_BYTES;
  static constexpr int DO_BYTES = (DV / 64) * QH_BYTES;
  static constexpr int PT_BYTES = HALF_BYTES;   // [128 kv x 64 q]
  static constexpr int SMEM = K_BYTES + V_BYTES + Q_BYTES + DO_BYTES + 2 * PT_BYTES + 1024 /*lse+delta*/ + 128 + 1024;
  static_assert(SMEM <= 227 * 1024, "");
  static constexpr int ST_COL = 0, DPT_COL = 64, DV_COL = 128, DK_COL = 256, DQ_COL = 384;
};

// Four softmax warpgroups share every q tile, 16 columns each: with nothing double-buffered (shared memory is full) an iteration
// is a chain of scores -> P^T, dS^T -> products, and more warps shorten its middle. lse / delta are requested two iterations early; dK
// comes first, so that Q, which the next scores wait for, loads beside dV and dQ^T; dO is handed back by itself; dQ^T has TMEM
// columns of its own, so that the next scores do not wait for its drain; tiles without a mask have a path of their own; and four rows
// of a dQ column lie side by side in the fp32 sum, which leaves in 16-byte reductions. 4 x 2048 tokens, 16 / 8 heads of 256, whole
// backward pass 904 -> 816 us, 300 + 2701 tokens 419 -> 378. Still the chain bounds it: the MMAs are a third of an iteration, half of
// it with their operand reads.
constexpr int WBWD_THREADS = 576;
template <int DQK, int DV, bool SOFTCAP>
__global__ void __launch_bounds__(WBWD_THREADS, 1)
    flash_wide_bwd_kernel(const __grid_constant__ CUtensorMap tm_kv, const __grid_constant__ CUtensorMap tm_q,
                          const __grid_constant__ CUtensorMap tm_do, const WideParams p) {
  using C = WBwd<DQK, DV>;
  const int tile_id = blockIdx.y;
  if (tile_id >= p.n_tiles) return;
  const int kv_head = blockIdx.x, part = blockIdx.z;
  const int group = p.Hq / p.Hk, head0 = kv_head * group;
  const int4 ti = p.tiles[tile_id];
  const int doc_start = ti.x, doc_len = ti.y, kv0 = ti.z;
  if (!AXB_INDEX_OK(AXB_SITE_ATTN_TILE, (long long)doc_start + doc_len - 1, p.T) || !AXB_INDEX_OK(AXB_SITE_ATTN_TILE, kv0, doc_len)) return;
  const bool bidir = ti.w & 1;
  const int win = bidir ? 0 : (ti.w >> 1);
  const int q_first = bidir ? 0 : kv0 / 64;
  int q_last = (doc_len + 63) / 64;
  if (win > 0) q_last = min(q_last, (kv0 + 127 + win - 1) / 64 + 1);
  const int n_qt = q_last - q_first;
  const int n_iter = n_qt * group;
  if (n_iter <= 0) return;
  // column parts of this CTA
  const bool has_k = part * 128 < DQK, has_v = part * 128 < DV;
  const int kpart = has_k ? min(part * 128, DQK - 128) : 0;   // first q/k column of the 128-wide window
  const int k_lo = has_k ? part * 128 - kpart : 128;          // columns of the window below k_lo belong to another part
  const int vpart = has_v ? part * 128 : 0;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::K_BYTES;
  uint8_t* sQ = sV + C::V_BYTES;
  uint8_t* sdO = sQ + C::Q_BYTES;
  uint8_t* sPT = sdO + C::DO_BYTES;
  uint8_t* sdST = sPT + C::PT_BYTES;
  float* s_rows = reinterpret_cast<float*>(sdST + C::PT_BYTES);  // per warpgroup: two buffers of -lse [16], -delta * scale [16]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_rows + 4 * 2 * 32);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;
  uint64_t* q_empty = bars + 2;
  uint64_t* s_full = bars + 3;
  uint64_t* pt_full = bars + 4;
  uint64_t* dq_full = bars + 5;
  uint64_t* st_free = bars + 6;
  uint64_t* acc_full = bars + 7;
  uint64_t* do_full = bars + 8;
  uint64_t* do_empty = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(pt_full, 512);
    mbar_init(dq_full, 1);
    mbar_init(st_free, 512);
    mbar_init(acc_full, 1);
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(kv_full, C::K_BYTES + C::V_BYTES);
#pragma unroll
      for (int h = 0; h < DQK / 64; ++h)
        tma_load_2d(sK + h * HALF_BYTES, &tm_kv, kv_full, p.k_col0 + kv_head * DQK + h * 64, doc_start + kv0);
#pragma unroll
      for (int h = 0; h < DV / 64; ++h)
        tma_load_2d(sV + h * HALF_BYTES, &tm_kv, kv_full, p.v_col0 + kv_head * DV + h * 64, doc_start + kv0);
    }
    __syncwarp();
    int qt = 0, head = head0;
    for (int it = 0; it < n_iter; ++it) {
      const int qrow = doc_start + (q_first + qt) * 64;
      if (!warp_all(mbar_wait(q_empty, (it & 1) ^ 1, p.status, AXB_TIMEOUT_EMPTY))) break;
      if (elect_one()) {
        mbar_expect_tx(q_full, C::Q_BYTES);
#pragma unroll
        for (int h = 0; h < DQK / 64; ++h)
          tma_load_2d(sQ + h * QH_BYTES, &tm_q, q_full, p.q_col0 + head * DQK + h * 64, qrow);
      }
      __syncwarp();
      if (!warp_all(mbar_wait(do_empty, (it & 1) ^ 1, p.status, AXB_TIMEOUT_EMPTY))) break;
      if (elect_one()) {
        mbar_expect_tx(do_full, C::DO_BYTES);
#pragma unroll
        for (int h = 0; h < DV / 64; ++h)
          tma_load_2d(sdO + h * QH_BYTES, &tm_do, do_full, head * DV + h * 64, qrow);
      }
      __syncwarp();
      if (++qt == n_qt) {
        qt = 0;
        ++head;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_st = make_idesc_bf16(128, 64, 0, 0);
    constexpr uint32_t idesc_acc = make_idesc_bf16(128, 128, 0, 1);
    constexpr uint32_t idesc_dq = make_idesc_bf16(128, 64, 1, 1);
    const uint64_t dk_k = make_smem_desc_sw128(smem_u32(sK), 16, 1024), dv_k = make_smem_desc_sw128(smem_u32(sV), 16, 1024);
    const uint64_t dq_k = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), do_k = make_smem_desc_sw128(smem_u32(sdO), 16, 1024);
    const uint64_t pt_k = make_smem_desc_sw128(smem_u32(sPT), 16, 1024), ds_k = make_smem_desc_sw128(smem_u32(sdST), 16, 1024);
    const uint64_t do_mn = make_smem_desc_sw128(smem_u32(sdO) + (vpart / 64) * QH_BYTES, QH_BYTES, 1024);
    const uint64_t dq_mn = make_smem_desc_sw128(smem_u32(sQ) + (kpart / 64) * QH_BYTES, QH_BYTES, 1024);
    const uint64_t dk_mn = make_smem_desc_sw128(smem_u32(sK) + (kpart / 64) * HALF_BYTES, HALF_BYTES, 1024);
    const uint64_t ds_mn = make_smem_desc_sw128(smem_u32(sdST), HALF_BYTES, 1024);
    bool ok = warp_all(mbar_wait(kv_full, 0, p.status, AXB_TIMEOUT_FULL));
    for (int it = 0; it < n_iter && ok; ++it) {
      const uint32_t ph = it & 1;
      if (!warp_all(mbar_wait(q_full, ph, p.status, AXB_TIMEOUT_FULL))) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < DQK / 16; ++kk) {
          const uint32_t koff = ((kk / 4) * HALF_BYTES + (kk % 4) * 32) / 16, qoff = ((kk / 4) * QH_BYTES + (kk % 4) * 32) / 16;
          umma_f16(tmem_base + C::ST_COL, dk_k + koff, dq_k + qoff, idesc_st, kk > 0);
        }
      }
      __syncwarp();
      if (!warp_all(mbar_wait(do_full, ph, p.status, AXB_TIMEOUT_FULL))) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < DV / 16; ++kk) {
          const uint32_t koff = ((kk / 4) * HALF_BYTES + (kk % 4) * 32) / 16, qoff = ((kk / 4) * QH_BYTES + (kk % 4) * 32) / 16;
          umma_f16(tmem_base + C::DPT_COL, dv_k + koff, do_k + qoff, idesc_st, kk > 0);
        }
        umma_commit(s_full);
      }
      __syncwarp();
      // dQ^T of the iteration before is out of its columns (long since), and P^T, dS^T of this one are in place
      bool fine = mbar_wait(pt_full, ph, p.status, AXB_TIMEOUT_GENERIC);
      if (fine && it > 0) fine = mbar_wait(st_free, (it - 1) & 1, p.status, AXB_TIMEOUT_TMEM_EMPTY);
      if (!warp_all(fine)) break;
      tc_fence_after();
      if (elect_one()) {
        if (has_k) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16(tmem_base + C::DK_COL, ds_k + kk * 2, dq_mn + kk * (2048 / 16), idesc_acc, (it > 0 || kk > 0));
        }
        umma_commit(q_empty);   // the next Q is the first that the next scores wait for: it loads beside dV and dQ^T
        if (has_v) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16(tmem_base + C::DV_COL, pt_k + kk * 2, do_mn + kk * (2048 / 16), idesc_acc, (it > 0 || kk > 0));
        }
        umma_commit(do_empty);
        if (has_k) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16(tmem_base + C::DQ_COL, dk_mn + kk * (2048 / 16), ds_mn + kk * (2048 / 16), idesc_dq, kk > 0);
        }
        umma_commit(dq_full);
        if (it == n_iter - 1) umma_commit(acc_full);
      }
      __syncwarp();
    }
  } else {
    const int lg = warp & 3;
    const int r = lg * 32 + lane;   // kv row of the tile (S^T, dP^T, dK, dV) or column of the part (dQ^T)
    const int grp = (warp - 2) >> 2, c0 = grp * 16;   // columns [c0, c0 + 16) of every q tile
    const int tid = threadIdx.x - 64 - grp * 128;
    const int kv_idx = kv0 + r;
    const uint32_t lane_off = uint32_t(lg * 32) << 16;
    float* const rows = s_rows + grp * 64;
    bool ok = true;
    // -lse or -delta * scale of one of this group's 16 q rows, requested two iterations ahead (rows outside: P = 0)
    auto fetch_row = [&](int it) -> float {
      float val = tid < 16 ? -INFINITY : 0.f;
      if (tid >= 32 || it >= n_iter) return val;
      const int q = (q_first + it % n_qt) * 64 + c0 + (tid & 15);
      const long long row = (long long)doc_start + q;
      if (q < doc_len && row < p.T) {
        const long long off = (long long)(head0 + it / n_qt) * p.T + row;
        val = tid < 16 ? -p.lse2[off] : -p.delta[off] * p.scale;
      }
      return val;
    };
    auto gradients = [&](auto masked, const uint32_t (&sr)[16], const uint32_t (&dr)[16], const float* nlse, int qc0, int q_lo, int q_hi) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t pk[4], dk[4];
#pragma unroll
        for (int i = q * 8; i < q * 8 + 8; i += 2) {
          float pv[2], dv[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float s = __uint_as_float(sr[i + e]);
            float g = 1.f;
            if constexpr (SOFTCAP) {
              const float t = tanhf(s * p.cap_in);
              pv[e] = fast_exp2(fmaf(t, p.cap_out2, nlse[i + e]));
              g = 1.f - t * t;
            } else {
              pv[e] = fast_exp2(fmaf(s, p.sl2, nlse[i + e]));
            }
            if (decltype(masked)::value && (qc0 + i + e < q_lo || qc0 + i + e > q_hi)) pv[e] = 0.f;
            dv[e] = pv[e] * fmaf(__uint_as_float(dr[i + e]), p.scale, nlse[16 + i + e]) * g;
          }
          pk[(i & 6) >> 1] = pack_bf16x2(pv[0], pv[1]);
          dk[(i & 6) >> 1] = pack_bf16x2(dv[0], dv[1]);
        }
        const uint32_t off = sw128_chunk_off(r, c0 / 8 + q);
        *reinterpret_cast<uint4*>(sPT + off) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(sdST + off) = make_uint4(dk[0], dk[1], dk[2], dk[3]);
      }
    };
    const long long width = (long long)p.Hq * DQK, rows4 = p.T & ~3ll;
    // the sums of 16 queries, the first one `shift` rows into its group of four; whole groups with 16-byte reductions
    auto add_rows = [&](auto shift, const uint32_t (&v)[16], float* to) {
      constexpr int a = decltype(shift)::value;
#pragma unroll
      for (int g = a ? 1 : 0; g < 4; ++g) red_add_f32x4(to + g * 4 * width, v[(4 * g - a) & 15], v[(4 * g - a + 1) & 15], v[(4 * g - a + 2) & 15], v[(4 * g - a + 3) & 15]);
      if (a == 1 || a == 3) red_add_f32(to + a, v[0]);
      if (a == 1 || a == 2) red_add_f32x2(to + 2, v[(2 - a) & 15], v[(3 - a) & 15]);
      if (a == 2 || a == 3) red_add_f32x2(to + 16 * width, v[(16 - a) & 15], v[(17 - a) & 15]);
      if (a == 1 || a == 3) red_add_f32(to + 16 * width + a - 1, v[15]);
    };
    float row_val = fetch_row(0);
    if (tid < 32) rows[tid] = row_val;
    row_val = fetch_row(1);
    asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
    for (int it = 0; it < n_iter; ++it) {
      const uint32_t ph = it & 1;
      const int head = head0 + it / n_qt;
      const int qc0 = (q_first + it % n_qt) * 64 + c0;      // doc-relative first q row of this group's columns
      // (a lane whose wait ran out walks on with the others, without waiting again: the group meets at the barrier below)
      ok = ok && mbar_wait(s_full, ph, p.status, AXB_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      const bool need_mask = (!bidir && qc0 < kv0 + 127) || kv0 + 128 > doc_len || (win > 0 && qc0 + 15 >= kv0 + win);
      {
        uint32_t sr[16], dr[16];
        tmem_ld_32x16(tmem_base + lane_off + C::ST_COL + c0, sr);
        tmem_ld_32x16(tmem_base + lane_off + C::DPT_COL + c0, dr);
        tmem_ld_wait();
        if (need_mask) {
          const bool row_in_doc = kv_idx < doc_len;
          const int q_lo = row_in_doc ? (bidir ? -(1 << 30) : kv_idx) : (1 << 30);
          const int q_hi = win > 0 ? kv_idx + win - 1 : (1 << 30);
          gradients(std::true_type{}, sr, dr, rows + ph * 32, qc0, q_lo, q_hi);
        } else {
          gradients(std::false_type{}, sr, dr, rows + ph * 32, 0, 0, 0);
        }
      }
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(pt_full);
      // lse / delta of the next iteration into the other buffer, while the MMAs run; the barrier also says that all warps of the group
      // have read the present one
      if (tid < 32) rows[(ph ^ 1) * 32 + tid] = row_val;
      row_val = fetch_row(it + 2);
      asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
      ok = ok && mbar_wait(dq_full, ph, p.status, AXB_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      if (has_k) {
        const long long row0 = (long long)doc_start + qc0;
        int i_hi = min(16, doc_len - qc0);
        if (row0 + i_hi > p.T) i_hi = (int)(p.T - row0);
        uint32_t qr[16];
        tmem_ld_32x16(tmem_base + lane_off + C::DQ_COL + c0, qr);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive(st_free);        // the next dQ^T may overwrite the columns while the sums leave
        if (r >= k_lo) {
          const long long col = (long long)head * DQK + kpart + r;
          if (((row0 + 15) | 3) < rows4) {      // every group of four rows that these touch is a whole one
            if (i_hi < 16) {
#pragma unroll
              for (int i = 0; i < 16; ++i) qr[i] = i < i_hi ? qr[i] : 0u;
            }
            float* to = p.dq_acc + (row0 & ~3ll) * width + col * 4;
            switch ((int)(row0 & 3)) {
              case 0: add_rows(std::integral_constant<int, 0>{}, qr, to); break;
              case 1: add_rows(std::integral_constant<int, 1>{}, qr, to); break;
              case 2: add_rows(std::integral_constant<int, 2>{}, qr, to); break;
              default: add_rows(std::integral_constant<int, 3>{}, qr, to); break;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (i < i_hi) atomicAdd(p.dq_acc + dq_at(row0 + i, col, width, rows4), __uint_as_float(qr[i]));
          }
        }
      } else {
        tc_fence_before();
        mbar_arrive(st_free);
      }
    }
    if (warp_all(ok && mbar_wait(acc_full, 0, p.status, AXB_TIMEOUT_TMEM_FULL))) {
      tc_fence_after();
      const bool row_ok = kv_idx < doc_len;
      const long long grow = (long long)doc_start + kv_idx;
      __nv_bfloat16* krow = p.dkv + grow * p.dkv_ld + p.dk_col0 + (long long)kv_head * DQK + kpart;
      __nv_bfloat16* vrow = p.dkv + grow * p.dkv_ld + p.dv_col0 + (long long)kv_head * DV + vpart;
      {
        const int c = grp;
        uint32_t a[32], b[32];
        tmem_ld_32x32(tmem_base + lane_off + C::DK_COL + c * 32, a);
        tmem_ld_32x32(tmem_base + lane_off + C::DV_COL + c * 32, b);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (has_k && c * 32 + q * 8 >= k_lo) {
              uint4 u;
              u.x = pack_bf16x2(__uint_as_float(a[q * 8 + 0]), __uint_as_float(a[q * 8 + 1]));
              u.y = pack_bf16x2(__uint_as_float(a[q * 8 + 2]), __uint_as_float(a[q * 8 + 3]));
              u.z = pack_bf16x2(__uint_as_float(a[q * 8 + 4]), __uint_as_float(a[q * 8 + 5]));
              u.w = pack_bf16x2(__uint_as_float(a[q * 8 + 6]), __uint_as_float(a[q * 8 + 7]));
              *reinterpret_cast<uint4*>(krow + c * 32 + q * 8) = u;
            }
            if (has_v) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(b[q * 8 + 0]), __uint_as_float(b[q * 8 + 1]));
              w.y = pack_bf16x2(__uint_as_float(b[q * 8 + 2]), __uint_as_float(b[q * 8 + 3]));
              w.z = pack_bf16x2(__uint_as_float(b[q * 8 + 4]), __uint_as_float(b[q * 8 + 5]));
              w.w = pack_bf16x2(__uint_as_float(b[q * 8 + 6]), __uint_as_float(b[q * 8 + 7]));
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
    tmem_dealloc(tmem_base, 512);
  }
}

template <int DQK, int DV, bool SC>
int launch_wide_fwd(const CUtensorMap& tq, const CUtensorMap& tkv, const WideParams& p, cudaStream_t st) {
  auto kern = flash_wide_fwd_kernel<DQK, DV, SC>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WFwd<DQK, DV>::SMEM);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  dim3 grid(p.Hq, p.n_tiles);
  kern<<<grid, 192, WFwd<DQK, DV>::SMEM, st>>>(tq, tkv, p);
  return (int)cudaGetLastError();
}
template <int DQK, int DV, bool SC>
int launch_wide_bwd(const CUtensorMap& tkv, const CUtensorMap& tq, const CUtensorMap& tdo, const WideParams& p,
                    cudaStream_t st) {
  using C = WBwd<DQK, DV>;
  auto kern = flash_wide_bwd_kernel<DQK, DV, SC>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  constexpr int pk = (DQK + 127) / 128, pv = (DV + 127) / 128;
  constexpr int parts = pk > pv ? pk : pv;
  dim3 grid(p.Hk, p.n_tiles, parts);
  kern<<<grid, WBWD_THREADS, C::SMEM, st>>>(tkv, tq, tdo, p);
  return (int)cudaGetLastError();
}

void fill_common(WideParams& p, const void* tiles, int n_tiles, int Hq, int Hk, int q_col0, int k_col0, int v_col0,
                 long long T, float scale, float softcap, int* status) {
  p.tiles = reinterpret_cast<const int4*>(tiles);
  p.n_tiles = n_tiles;
  p.Hq = Hq;
  p.Hk = Hk;
  p.q_col0 = q_col0;
  p.k_col0 = k_col0;
  p.v_col0 = v_col0;
  p.T = T;
  p.scale = scale;
  p.sl2 = scale * 1.4426950408889634f;
  p.cap_in = softcap > 0.f ? scale / softcap : 0.f;
  p.cap_out2 = softcap * 1.4426950408889634f;
  p.status = status;
}

}  // namespace

// qkv [T, Hq*Dqk | Hk*Dqk | Hk*Dv] bf16 (column offsets given), out [T, Hq*Dv], lse2 [Hq, T] fp32.
// (Dqk, Dv) in {(256, 256), (192, 128)}; softcap 0 = none.
extern "C" int axb_flash_wide_fwd(const void* qkv, long long ld, long long T, int Hq, int Hk, int Dqk, int Dv,
                                  int q_col0, int k_col0, int v_col0, const void* tiles, int n_tiles, void* out,
                                  long long out_ld, float* lse2, float softmax_scale, float softcap, int* status,
                                  void* stream) {
  if (T <= 0 || n_tiles <= 0) return 0;
  if (!((Dqk == 256 && Dv == 256) || (Dqk == 192 && Dv == 128))) return -2;
  if ((ld & 7) || (out_ld & 7) || (q_col0 & 7) || (k_col0 & 7) || (v_col0 & 7) || Hk <= 0 || Hq % Hk) return -3;
  CUtensorMap tq;
  if (axb_make_tmap_2d(&tq, qkv, T, ld, ld, 128, 64)) return -4;
  WideParams p = {};
  fill_common(p, tiles, n_tiles, Hq, Hk, q_col0, k_col0, v_col0, T, softmax_scale, softcap, status);
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.out_ld = out_ld;
  p.lse2 = lse2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool sc = softcap > 0.f;
  if (Dqk == 256) return sc ? launch_wide_fwd<256, 256, true>(tq, tq, p, st) : launch_wide_fwd<256, 256, false>(tq, tq, p, st);
  return sc ? launch_wide_fwd<192, 128, true>(tq, tq, p, st) : launch_wide_fwd<192, 128, false>(tq, tq, p, st);
}

// dout / out [T, Hq*Dv] (ld o_ld); dqkv same layout as qkv; dq_acc fp32 [T, Hq*Dqk] and delta fp32 [Hq, T] scratch.
extern "C" int axb_flash_wide_bwd(const void* qkv, long long ld, const void* dout, const void* out, long long o_ld,
                                  const float* lse2, long long T, int Hq, int Hk, int Dqk, int Dv, int q_col0,
                                  int k_col0, int v_col0, const void* tiles, int n_tiles, void* dqkv,
                                  long long dqkv_ld, float* dq_acc, float* delta, float softmax_scale, float softcap,
                                  int* status, void* stream) {
  if (T <= 0 || n_tiles <= 0) return 0;
  if (!((Dqk == 256 && Dv == 256) || (Dqk == 192 && Dv == 128))) return -2;
  if ((ld & 7) || (o_ld & 7) || (dqkv_ld & 7) || (q_col0 & 7) || (k_col0 & 7) || (v_col0 & 7) || Hk <= 0 || Hq % Hk) return -3;
  if (!attn_bwd_aligned(out, dqkv, dq_acc)) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap tkv, tq, tdo;
  if (axb_make_tmap_2d(&tkv, qkv, T, ld, ld, 128, 64)) return -4;
  if (axb_make_tmap_2d(&tq, qkv, T, ld, ld, 64, 64)) return -4;
  if (axb_make_tmap_2d(&tdo, dout, T, (long long)Hq * Dv, o_ld, 64, 64)) return -4;
  cudaError_t e = cudaMemsetAsync(dq_acc, 0, sizeof(float) * T * Hq * Dqk, st);
  if (e != cudaSuccess) return (int)e;
  if (Dv == 256) launch_attn_delta<256>(dout, out, delta, T, Hq, o_ld, st);
  else launch_attn_delta<128>(dout, out, delta, T, Hq, o_ld, st);
  WideParams p = {};
  fill_common(p, tiles, n_tiles, Hq, Hk, q_col0, k_col0, v_col0, T, softmax_scale, softcap, status);
  p.lse2 = const_cast<float*>(lse2);
  p.delta = delta;
  p.dq_acc = dq_acc;
  p.dkv = reinterpret_cast<__nv_bfloat16*>(dqkv);
  p.dkv_ld = dqkv_ld;
  p.dk_col0 = k_col0;
  p.dv_col0 = v_col0;
  const bool sc = softcap > 0.f;
  int rc;
  if (Dqk == 256) rc = sc ? launch_wide_bwd<256, 256, true>(tkv, tq, tdo, p, st) : launch_wide_bwd<256, 256, false>(tkv, tq, tdo, p, st);
  else rc = sc ? launch_wide_bwd<192, 128, true>(tkv, tq, tdo, p, st) : launch_wide_bwd<192, 128, false>(tkv, tq, tdo, p, st);
  if (rc) return rc;
  launch_dq_convert(dq_acc, dqkv, T, Hq * Dqk, dqkv_ld, q_col0, st);
  return (int)cudaGetLastError();
}
