// Single-query (decode) attention over a per-sequence KV cache for sm_100a.
//
// Bound: one pass over the live part of the cache (HBM). Everything else is arranged so that enough bytes are in
// flight: the positions of one (sequence, kv head) are split over a thread-block cluster of up to 8 CTAs of four
// warps, and every warp streams its own 16-position K / V tiles through a private ring of cp.async stages (no CTA
// barrier in the loop; two CTAs per SM keep about 130 KB in flight at D = 128). The whole GQA group of query heads is
// served from one read of the cache: up to 16 heads are the 16 rows of mma.sync m16n8k16 tiles, whose rate is four
// times what the stream needs (a 128-row tcgen05 tile would be 7/8 padding). Scores, softmax statistics and sums are
// fp32; probabilities enter the second product as hi + lo bf16 pairs (16 significant bits), so that splitting them for
// the tensor cores adds less than 2^-16 to a result that is rounded to bf16.
// The partial results of a cluster meet in distributed shared memory: no workspace, no second launch, fixed order.
// Measured (one layer, 32 q / 8 kv heads of 128, L2 flushed): 64 sequences of 500 to 4096 positions 142 us = 4.6 TB/s
// (1148 us with one CTA per pair scoring one position per thread), 8 sequences of 200 to 900 positions 19 us (234 us).
//
// Optional, for a generation step: the kernel rotates q and the new k itself (rotary embedding, `inv_freq` != null) and
// appends the new k / v row to the cache (`append`). Only cluster rank 0 stores the row; the warp whose tile holds the
// new position takes it from shared memory, so no CTA waits for another one's store. Row and position are compared with the
// cache's: a sequence outside it gets zeros, stores nothing and is reported through the status word.
//
// Generation in the reference goes through Hugging Face `generate` with its KV cache and SDPA /
// flash-attn decode kernels (src/axolotl/cli/inference.py, core/trainers/grpo rollouts).
#include "axb_common.cuh"

namespace {

constexpr int DEC_W = 4;            // warps per CTA
constexpr int DEC_T = 32 * DEC_W;
constexpr int MAX_G = 16;           // query heads per kv head (rows of the MMA tile)
constexpr int DEC_P = 16;           // positions per warp tile
constexpr int DEC_MAX_SPLITS = 8;   // portable cluster size

struct DecodeParams {
  const __nv_bfloat16* qkv;
  long long ld;
  int q_col0, k_col0, v_col0;       // k_col0 / v_col0: columns of the new token's k / v (append only)
  __nv_bfloat16* kc;
  __nv_bfloat16* vc;
  const long long* seq;             // cache row of every query row, or null (row b uses cache row b)
  const int* lens;                  // live positions including the new token
  const int* pos;                   // rotary positions
  const float* inv_freq;            // null: q and k are rotated already
  float attn_scale;
  __nv_bfloat16* out;
  long long out_ld;
  int Hq, Hk;
  long long max_len, rows;          // positions per cache row, cache rows
  float scale;
  int window;
  int append;
  int* status;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// pair (x, y) as hi + lo bf16 pairs
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16x2(x, y);
  const float2 h = unpack_bf16x2(hi);
  lo = pack_bf16x2(x - h.x, y - h.y);
}
template <int D>
struct DecCfg {
  static constexpr int ROWB = D * 2;                       // bytes of one cache row of a head
  static constexpr int CH = D / 8;                         // 16-byte chunks per row
  static constexpr int TILE = DEC_P * ROWB;                // K (or V) part of a stage
  static constexpr int STAGES = D == 64 ? 4 : (D == 128 ? 3 : 2);
  static constexpr int RING = DEC_W * STAGES * 2 * TILE;   // D = 128: 96 KB (two CTAs per SM)
  static constexpr int Q_BYTES = MAX_G * ROWB;
  static constexpr int NEW_BYTES = 2 * ROWB;
  static constexpr int STAT = DEC_W * MAX_G;               // per-warp row statistics
  static constexpr int SMEM = RING + Q_BYTES + NEW_BYTES + (2 * STAT + 2 * DEC_MAX_SPLITS * STAT) * 4 + D * 4;
};

template <int D>
__global__ void __launch_bounds__(DEC_T) decode_attn_kernel(const DecodeParams p) {
  using C = DecCfg<D>;
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t* ring = smem;
  uint8_t* sQ = smem + C::RING;
  uint8_t* sNew = sQ + C::Q_BYTES;                         // rotated k row, v row of the new token
  float* sM = reinterpret_cast<float*>(sNew + C::NEW_BYTES);
  float* sL = sM + C::STAT;
  float* gM = sL + C::STAT;                                // statistics of all warps of the cluster, then weights
  float* gL = gM + DEC_MAX_SPLITS * C::STAT;
  float* sCS = gL + DEC_MAX_SPLITS * C::STAT;              // cos | sin of the new position
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch_dependents();
  const int kvh = blockIdx.y, b = blockIdx.z;
  const int rank = (int)cluster_ctarank(), nsplit = (int)cluster_nctarank();
  const int G = p.Hq / p.Hk;
  int n = p.lens[b];
  long long crow = p.seq ? p.seq[b] : (long long)b, at = n - 1;      // cache row, position of the new token
  if (crow < 0) crow += p.rows;                            // counted from the end, as an indexed store does
  if (at < 0 && p.append) at += p.max_len;
  if (!axb_index_checked(AXB_SITE_CACHE_ROW, crow, p.rows, tid == 0 && kvh == 0 && rank == 0, p.status) ||
      !axb_index_checked(AXB_SITE_CACHE_POS, max(at, p.append ? at : 0ll), p.max_len, tid == 0 && kvh == 0 && rank == 0, p.status)) {
    n = 0;                                                 // nothing is read or stored, the result is zero
    at = -1;
  }
  const int first = p.window > 0 ? max(0, n - p.window) : 0;
  const int n_load = p.append ? n - 1 : n;                 // the appended row comes from shared memory
  const long long row_elems = (long long)p.Hk * D;
  __nv_bfloat16* kb = p.kc + crow * p.max_len * row_elems + (long long)kvh * D;
  __nv_bfloat16* vb = p.vc + crow * p.max_len * row_elems + (long long)kvh * D;
  const int tiles = n > first ? (n - first + DEC_P - 1) / DEC_P : 0;
  const int step = nsplit * DEC_W;
  const uint32_t wring = smem_u32(ring) + warp * (C::STAGES * 2 * C::TILE);

  auto load_tile = [&](int tile, int stage) {
    if (tile < tiles) {
      const uint32_t dst = wring + stage * 2 * C::TILE;
      const int p0 = first + tile * DEC_P;
#pragma unroll
      for (int i = 0; i < DEC_P * C::CH / 32; ++i) {
        const int idx = lane + 32 * i;
        const int row = idx / C::CH, ch = idx % C::CH;
        const bool ok = p0 + row < n_load;
        const long long off = ok ? (long long)(p0 + row) * row_elems + ch * 8 : 0;
        const uint32_t d = dst + row * C::ROWB + ((ch ^ (row & 7)) << 4);
        cp_async16(d, kb + off, ok ? 16 : 0);              // rows past the end read as zeros
        cp_async16(d + C::TILE, vb + off, ok ? 16 : 0);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int tile = rank * DEC_W + warp;
#pragma unroll
  for (int s = 0; s < C::STAGES - 1; ++s) load_tile(tile + s * step, s);

  pdl_wait();            // the rows of the cache above are older than the kernel this launch may overlap; qkv is not

  // ---- query rows (and the new k / v row), rotated on the way when asked
  const __nv_bfloat16* qrow = p.qkv + (long long)b * p.ld;
  if (p.inv_freq) {
    const float ps = (float)p.pos[b];
    for (int j = tid; j < D / 2; j += DEC_T) {
      float s, c;
      sincosf(ps * p.inv_freq[j], &s, &c);
      sCS[j] = c * p.attn_scale;
      sCS[D / 2 + j] = s * p.attn_scale;
    }
    __syncthreads();
  }
  for (int i = tid; i < (MAX_G + 1) * (D / 2); i += DEC_T) {
    const int g = i / (D / 2), j = i % (D / 2);
    if (g == MAX_G && !p.append) continue;
    float a = 0.f, c = 0.f;
    if (g < G || g == MAX_G) {
      const __nv_bfloat16* src = qrow + (g == MAX_G ? p.k_col0 + kvh * D : p.q_col0 + (kvh * G + g) * D);
      a = __bfloat162float(src[j]);
      c = __bfloat162float(src[j + D / 2]);
      if (p.inv_freq) {
        const float cs = sCS[j], sn = sCS[D / 2 + j], a0 = a;
        a = a0 * cs - c * sn;
        c = c * cs + a0 * sn;
      }
    }
    if (g == MAX_G) {
      reinterpret_cast<__nv_bfloat16*>(sNew)[j] = __float2bfloat16(a);
      reinterpret_cast<__nv_bfloat16*>(sNew)[j + D / 2] = __float2bfloat16(c);
    } else {
      auto put = [&](int d, float v) {
        *reinterpret_cast<__nv_bfloat16*>(sQ + g * C::ROWB + ((((d >> 3) ^ (g & 7))) << 4) + (d & 7) * 2) = __float2bfloat16(v);
      };
      put(j, a);
      put(j + D / 2, c);
    }
  }
  if (p.append)
    for (int j = tid; j < D; j += DEC_T) reinterpret_cast<__nv_bfloat16*>(sNew)[D + j] = qrow[p.v_col0 + kvh * D + j];
  __syncthreads();
  if (p.append && rank == 0 && at >= 0) {
    for (int j = tid; j < D; j += DEC_T) {
      kb[at * row_elems + j] = reinterpret_cast<const __nv_bfloat16*>(sNew)[j];
      vb[at * row_elems + j] = reinterpret_cast<const __nv_bfloat16*>(sNew)[D + j];
    }
  }

  const int mi = lane >> 3, mr = lane & 7;
  const uint32_t q_base = smem_u32(sQ);
  // A operand (16 heads x 16 dims): matrices (rows 0-7, k 0-7), (rows 8-15, k 0-7), (rows 0-7, k 8-15), (rows 8-15, k 8-15)
  auto load_q = [&](int ks, uint32_t (&r)[4]) {
    const int row = (mi & 1) * 8 + mr, ch = ks * 2 + (mi >> 1);
    ldsm4(q_base + row * C::ROWB + ((ch ^ (row & 7)) << 4), r);
  };
  constexpr bool Q_REGS = D <= 128;
  uint32_t qf[Q_REGS ? D / 16 : 1][4];
  if (Q_REGS) {
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) load_q(ks, qf[Q_REGS ? ks : 0]);
  }
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  const float sc = p.scale * 1.4426950408889634f;
  int stage = 0;
  for (; tile < tiles; tile += step) {
    const int nst = stage == 0 ? C::STAGES - 1 : stage - 1;    // stage consumed in the previous iteration
    load_tile(tile + (C::STAGES - 1) * step, nst);
    cp_async_wait<C::STAGES - 1>();
    __syncwarp();
    const uint32_t kt = wring + stage * 2 * C::TILE, vt = kt + C::TILE;
    const int p0 = first + tile * DEC_P;
    if (p.append && p0 + DEC_P >= n) {                          // the tile of the new position
      const int row = n - 1 - p0;
      for (int ch = lane; ch < C::CH; ch += 32) {
        const uint32_t off = warp * (C::STAGES * 2 * C::TILE) + stage * 2 * C::TILE + row * C::ROWB + ((ch ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(ring + off) = *reinterpret_cast<const uint4*>(sNew + ch * 16);
        *reinterpret_cast<uint4*>(ring + off + C::TILE) = *reinterpret_cast<const uint4*>(sNew + C::ROWB + ch * 16);
      }
      __syncwarp();
    }
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t kf[4], qt[4];
      const int row = (mi >> 1) * 8 + mr, ch = ks * 2 + (mi & 1);
      ldsm4(kt + row * C::ROWB + ((ch ^ (row & 7)) << 4), kf);
      if (!Q_REGS) load_q(ks, qt);
      mma16816(s[0], Q_REGS ? qf[Q_REGS ? ks : 0] : qt, kf[0], kf[1]);
      mma16816(s[1], Q_REGS ? qf[Q_REGS ? ks : 0] : qt, kf[2], kf[3]);
    }
    // this lane: heads lane/4 and lane/4 + 8, positions p0 + 8 * t + 2 * (lane % 4) + {0, 1}
#pragma unroll
    for (int t = 0; t < 2; ++t) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int ps = p0 + t * 8 + 2 * (lane & 3) + (e & 1);
        s[t][e] = ps < n ? s[t][e] * sc : -INFINITY;
      }
    }
    float x0 = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
    float x1 = fmaxf(fmaxf(s[0][2], s[0][3]), fmaxf(s[1][2], s[1][3]));
    x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1));
    x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2));
    const float m0_old = m0, m1_old = m1;
    m0 = fmaxf(m0, x0);
    m1 = fmaxf(m1, x1);
    const float b0 = m0 == -INFINITY ? 0.f : m0, b1 = m1 == -INFINITY ? 0.f : m1;    // no finite score so far: every P is 0
    const float a0 = exp2f(m0_old - b0), a1 = exp2f(m1_old - b1);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      s[t][0] = exp2f(s[t][0] - b0);
      s[t][1] = exp2f(s[t][1] - b0);
      s[t][2] = exp2f(s[t][2] - b1);
      s[t][3] = exp2f(s[t][3] - b1);
    }
    l0 = l0 * a0 + ((s[0][0] + s[0][1]) + (s[1][0] + s[1][1]));
    l1 = l1 * a1 + ((s[0][2] + s[0][3]) + (s[1][2] + s[1][3]));
    uint32_t ph[4], pl[4];
    split_pair(s[0][0], s[0][1], ph[0], pl[0]);
    split_pair(s[0][2], s[0][3], ph[1], pl[1]);
    split_pair(s[1][0], s[1][1], ph[2], pl[2]);
    split_pair(s[1][2], s[1][3], ph[3], pl[3]);
#pragma unroll
    for (int i = 0; i < D / 16; ++i) {
      uint32_t vf[4];
      const int row = (mi & 1) * 8 + mr, ch = i * 2 + (mi >> 1);
      ldsm4_t(vt + row * C::ROWB + ((ch ^ (row & 7)) << 4), vf);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float(&oo)[4] = o[2 * i + h];
        oo[0] *= a0;
        oo[1] *= a0;
        oo[2] *= a1;
        oo[3] *= a1;
        mma16816(oo, ph, vf[2 * h], vf[2 * h + 1]);
        mma16816(oo, pl, vf[2 * h], vf[2 * h + 1]);
      }
    }
    __syncwarp();                                              // the stage is free for the next load
    stage = stage + 1 == C::STAGES ? 0 : stage + 1;
  }
  cp_async_wait<0>();
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
  l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const int r0 = lane >> 2, r1 = r0 + 8;
  if ((lane & 3) == 0) {
    sM[warp * MAX_G + r0] = m0;
    sM[warp * MAX_G + r1] = m1;
    sL[warp * MAX_G + r0] = l0;
    sL[warp * MAX_G + r1] = l1;
  }
  __syncthreads();                                             // every warp has left the ring: partial outputs go there
  float* part = reinterpret_cast<float*>(ring);                // [DEC_W][G][D]
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    const int d = i * 8 + 2 * (lane & 3);
    if (r0 < G) *reinterpret_cast<float2*>(part + ((long long)warp * G + r0) * D + d) = make_float2(o[i][0], o[i][1]);
    if (r1 < G) *reinterpret_cast<float2*>(part + ((long long)warp * G + r1) * D + d) = make_float2(o[i][2], o[i][3]);
  }
  cluster_sync();
  const int nw = nsplit * DEC_W;
  for (int i = tid; i < nw * MAX_G; i += DEC_T) {
    const int src = i / C::STAT, off = i % C::STAT;
    gM[i] = ld_cluster_f32(mapa_u32(smem_u32(sM + off), src));
    gL[i] = ld_cluster_f32(mapa_u32(smem_u32(sL + off), src));
  }
  __syncthreads();
  if (tid < G) {
    float mg = -INFINITY, lg = 0.f;
    for (int w = 0; w < nw; ++w) mg = fmaxf(mg, gM[w * MAX_G + tid]);
    for (int w = 0; w < nw; ++w) {                             // warps without a tile: m = -inf, weight 0
      const float f = gM[w * MAX_G + tid] == -INFINITY ? 0.f : exp2f(gM[w * MAX_G + tid] - mg);
      lg += f * gL[w * MAX_G + tid];
      gM[w * MAX_G + tid] = f;
    }
    gL[tid] = n > 0 ? 1.f / lg : 0.f;
  }
  __syncthreads();
  const uint32_t part_base = smem_u32(part);
  for (int i = rank * DEC_T + tid; i < G * (D / 4); i += nsplit * DEC_T) {
    const int g = i / (D / 4), d = (i % (D / 4)) * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int w = 0; w < nw; ++w) {
      const float f = gM[w * MAX_G + g];
      const float4 v = ld_cluster_f32x4(mapa_u32(part_base + (((w % DEC_W) * G + g) * D + d) * 4, w / DEC_W));
      acc.x += f * v.x;
      acc.y += f * v.y;
      acc.z += f * v.z;
      acc.w += f * v.w;
    }
    const float inv = gL[g];
    __nv_bfloat16* orow = p.out + (long long)b * p.out_ld + (long long)(kvh * G + g) * D + d;
    orow[0] = __float2bfloat16(acc.x * inv);
    orow[1] = __float2bfloat16(acc.y * inv);
    orow[2] = __float2bfloat16(acc.z * inv);
    orow[3] = __float2bfloat16(acc.w * inv);
  }
  cluster_sync();                                              // peers may still read this CTA's partial results
}

template <int D>
int launch_decode(const DecodeParams& p, int B, int splits, bool pdl, cudaStream_t st) {
  using C = DecCfg<D>;
  auto kern = decode_attn_kernel<D>;
  static std::atomic<unsigned long long> allowed{0};
  if (const int rc = axb_allow_smem((const void*)kern, C::SMEM, allowed)) return rc;
  AxbLaunch l(dim3((unsigned)splits, (unsigned)p.Hk, (unsigned)B), DEC_T, C::SMEM, st, splits, pdl);
  const cudaError_t e = cudaLaunchKernelEx(&l.cfg, kern, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// CTAs per (sequence, kv head). Splitting pays until the pairs fill the chip about once (two CTAs per SM): 16 x 8 pairs of
// 4000 positions took 72.7 / 64.5 / 69.7 / 90.1 us with 1 / 2 / 4 / 8 CTAs, 8 x 8 pairs of 30000 took 466 / 242 / 177 /
// 189 us (L2 flushed); beyond that the merge costs more than it brings. Batches with more pairs still take two, because
// their sequences differ in length and shorter CTAs even that out (64 x 8 pairs of 500 to 4096 positions: 162 / 142 /
// 154 us), unless there are many waves anyway. Never less than one tile per warp at the cache's capacity.
int pick_splits(int B, int Hk, long long max_len) {
  const long long pairs = (long long)B * Hk;
  int s = 1;
  while (s < DEC_MAX_SPLITS && (pairs * s < 256 || (s == 1 && pairs < 1024)) && (long long)s * 2 * DEC_W * DEC_P <= max_len) s *= 2;
  return s;
}

// Prompt rows into the cache: row t of the k and v blocks goes to (seq[t], pos[t]). One warp per row and block.
// Bound: HBM, twice the rows' bytes. 16-byte accesses: 6.4 us for 4096 rows of 2 x 1024, against 65 us for two indexed stores.
__global__ void __launch_bounds__(256) kv_append_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld, int k_col0, int v_col0,
                                                        __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc,
                                                        const long long* __restrict__ seq, const long long* __restrict__ pos, int T,
                                                        int width, long long rows, long long max_len, int* status) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long t = w >> 1;
  if (t >= T) return;
  long long b = seq[t], i = pos[t];
  if (b < 0) b += rows;                        // counted from the end, as an indexed store does
  if (i < 0) i += max_len;
  const bool report = lane == 0 && !(w & 1);
  if (!axb_index_checked(AXB_SITE_CACHE_ROW, b, rows, report, status) || !axb_index_checked(AXB_SITE_CACHE_POS, i, max_len, report, status))
    return;
  const __nv_bfloat16* src = qkv + t * ld + ((w & 1) ? v_col0 : k_col0);
  __nv_bfloat16* dst = ((w & 1) ? vc : kc) + (b * max_len + i) * width;
#pragma unroll 4
  for (int c = lane * 8; c < width; c += 256) *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
}

}  // namespace

// k_cache / v_cache [rows, max_len, width]; all rows 16-byte aligned, width a multiple of 8. A row outside [-rows, rows) or a
// position outside [-max_len, max_len) is not stored and sets *status (null: not reported).
extern "C" int axb_cache_append(const void* qkv, long long ld, int k_col0, int v_col0, void* k_cache, void* v_cache,
                                const long long* seq, const long long* pos, int T, int width, long long rows, long long max_len,
                                int* status, void* stream) {
  if (T <= 0) return 0;
  if ((ld & 7) || (k_col0 & 7) || (v_col0 & 7) || (width & 7)) return -2;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) return -3;
  kv_append_kernel<<<(unsigned)(((long long)T * 2 + 7) / 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      (const __nv_bfloat16*)qkv, ld, k_col0, v_col0, (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, seq, pos, T, width, rows, max_len,
      status);
  return (int)cudaGetLastError();
}
extern "C" int axb_kv_append(const void* qkv, long long ld, int k_col0, int v_col0, void* k_cache, void* v_cache, const long long* seq,
                             const long long* pos, int T, int width, long long rows, long long max_len, void* stream) {
  return axb_cache_append(qkv, ld, k_col0, v_col0, k_cache, v_cache, seq, pos, T, width, rows, max_len, nullptr, stream);
}

// qkv: [B, ld] fused projection of the new tokens (q block at column q_col0; rotated already unless inv_freq is given);
// k_cache / v_cache: [rows, max_len, Hk*D], 16-byte aligned; row b uses cache row seq[b] (seq == null: row b);
// lens[b]: live positions of sequence b including the new token; out: [B, out_ld >= Hq*D].
// append: the new token's k / v (columns k_col0 / v_col0 of qkv) are stored at position lens[b] - 1 and attended to;
// otherwise that position is read from the cache. inv_freq [D/2] + pos [B]: q (and the appended k) are rotated here.
// splits: 0 = chosen by pick_splits. pdl: the launch may overlap the end of its predecessor on the stream, which must not
// write the caches or lens. A cache row outside [-rows, rows) or a length above max_len sets *status (null: not reported).
extern "C" int axb_cache_attend(const void* qkv, long long ld, int q_col0, int k_col0, int v_col0, void* k_cache, void* v_cache,
                                long long rows, const long long* seq, const int* lens, const int* pos, const float* inv_freq,
                                float attn_scale, void* out, long long out_ld, int B, int Hq, int Hk, int D, long long max_len,
                                float scale, int window, int append, int splits, int pdl, int* status, void* stream) {
  if (B <= 0) return 0;
  if (Hk <= 0 || Hq % Hk || Hq / Hk > MAX_G || B > 65535) return -2;
  if ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) return -3;
  if (splits < 0 || splits > DEC_MAX_SPLITS) return -2;
  DecodeParams p;
  p.qkv = (const __nv_bfloat16*)qkv;
  p.ld = ld;
  p.q_col0 = q_col0;
  p.k_col0 = k_col0;
  p.v_col0 = v_col0;
  p.kc = (__nv_bfloat16*)k_cache;
  p.vc = (__nv_bfloat16*)v_cache;
  p.seq = seq;
  p.lens = lens;
  p.pos = pos;
  p.inv_freq = inv_freq;
  p.attn_scale = attn_scale;
  p.out = (__nv_bfloat16*)out;
  p.out_ld = out_ld;
  p.Hq = Hq;
  p.Hk = Hk;
  p.max_len = max_len;
  p.rows = rows;
  p.scale = scale;
  p.window = window;
  p.append = append;
  p.status = status;
  if (splits == 0) splits = pick_splits(B, Hk, max_len);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (D == 64) return launch_decode<64>(p, B, splits, pdl != 0, st);
  if (D == 128) return launch_decode<128>(p, B, splits, pdl != 0, st);
  if (D == 256) return launch_decode<256>(p, B, splits, pdl != 0, st);
  return -2;
}

// The same for a cache of B rows.
extern "C" int axb_decode_attn(const void* qkv, long long ld, int q_col0, int k_col0, int v_col0, void* k_cache, void* v_cache,
                               const long long* seq, const int* lens, const int* pos, const float* inv_freq, float attn_scale,
                               void* out, long long out_ld, int B, int Hq, int Hk, int D, long long max_len, float scale,
                               int window, int append, int splits, int pdl, void* stream) {
  return axb_cache_attend(qkv, ld, q_col0, k_col0, v_col0, k_cache, v_cache, B, seq, lens, pos, inv_freq, attn_scale, out, out_ld, B,
                          Hq, Hk, D, max_len, scale, window, append, splits, pdl, nullptr, stream);
}
