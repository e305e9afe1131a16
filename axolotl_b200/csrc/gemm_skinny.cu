// GEMM with one long and one short side, for sm_100a: acc[r, n] = sum_k P[r, k] S[n, k] (+ P2 S2^T), N <= 128
// (up to 256 as two launches).
//
//   out_mode 0: C[n, r]  (a generation step or a short row: P = weight, S = tokens, y = x W^T)
//   out_mode 1: C[r, n]  (the low-rank product x A^T of an adapter: P = tokens, S = A)
//   out_mode 2: h[n, r] = act(gate) * up with P = gate | up rows [2I, K]: a tile is 64 gate rows and the 64 up rows of the
//               same columns, so that the gated activation needs no pass of its own
//
// Bound: one pass over P (HBM). The long side is the 128-row operand of tcgen05.mma, so no tensor-core row is padding and the
// short side is the MMA's N = 16 .. 128; a 128 x 128-tile kernel reads the same bytes with only R / 128 CTAs, too few to keep
// HBM busy. Here the K range of a tile is split over a cluster of up to 8 CTAs and two CTAs share an SM, so that about 200 KB
// per SM are in flight; the partial tiles meet in distributed shared memory in a fixed order (no atomics, no workspace).
// In a dependent launch the tiles of P (a weight) are requested before the predecessor has finished.
#include "axb_common.cuh"

namespace {

constexpr int SK_T = 128;
constexpr int SK_BM = 128;
constexpr int SK_BK = 64;
constexpr int SK_P_BYTES = SK_BM * SK_BK * 2;

struct SkinnyParams {
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;   // added per P row (out_mode 0)
  int R, N, K, K2;             // out_mode 2: R counts the I columns of h
  float alpha;
  int out_mode, out_f32, p_dep;
  int glu_kind;
  float glu_limit;
  int* status;
};

template <int NT>
struct SkCfg {
  static constexpr int S_BYTES = NT * SK_BK * 2;
  static constexpr int STAGE = SK_P_BYTES + S_BYTES;
  static constexpr int STAGES = NT <= 32 ? 5 : (NT == 64 ? 4 : 3);
  static constexpr int RING = STAGES * STAGE;      // 84 .. 100 KB
  static constexpr int SMEM = RING + 1024 + 256;
  static constexpr int TMEM_COLS = NT < 32 ? 32 : NT;
  static_assert(NT * SK_BM * 4 <= RING, "the partial tile reuses the ring");
};

__device__ __forceinline__ float sk_act(float g, int kind) {
  if (kind == 0) return g * __fdividef(1.f, 1.f + __expf(-g));
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * g * (1.f + tanhf(k0 * (g + k1 * g * g * g)));
}

template <int NT>
__global__ void __launch_bounds__(SK_T)
    gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmS,
                       const __grid_constant__ CUtensorMap tmP2, const __grid_constant__ CUtensorMap tmS2, const SkinnyParams p) {
  using C = SkCfg<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::RING);
  uint64_t* empty = full + C::STAGES;
  uint64_t* done = empty + C::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int rank = (int)cluster_ctarank(), cs = (int)cluster_nctarank();
  const int tile = blockIdx.x / cs;
  const bool glu = p.out_mode == 2;
  const int nk_main = (p.K + SK_BK - 1) / SK_BK, nk = nk_main + (p.K2 + SK_BK - 1) / SK_BK;
  const int kb0 = (int)((long long)nk * rank / cs), kb1 = (int)((long long)nk * (rank + 1) / cs);

  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmP);
    tma_prefetch_desc(&tmS);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    auto load_p = [&](int kb, int s) {
      const bool ext = kb >= nk_main;
      const int k0 = (ext ? kb - nk_main : kb) * SK_BK;
      uint8_t* dst = smem + s * C::STAGE;
      const CUtensorMap* m = ext ? &tmP2 : &tmP;
      if (glu) {
        tma_load_2d(dst, m, &full[s], k0, tile * 64);
        tma_load_2d(dst + SK_P_BYTES / 2, m, &full[s], k0, p.R + tile * 64);
      } else {
        tma_load_2d(dst, m, &full[s], k0, tile * SK_BM);
      }
    };
    auto load_s = [&](int kb, int s) {
      const bool ext = kb >= nk_main;
      tma_load_2d(smem + s * C::STAGE + SK_P_BYTES, ext ? &tmS2 : &tmS, &full[s], (ext ? kb - nk_main : kb) * SK_BK, 0);
    };
    if (p.p_dep) pdl_wait();
    const int pre = min(C::STAGES, kb1 - kb0);
    for (int i = 0; i < pre; ++i) {
      if (elect_one()) {
        mbar_expect_tx(&full[i], C::STAGE);
        load_p(kb0 + i, i);
      }
      __syncwarp();
    }
    pdl_wait();
    for (int i = 0; i < pre; ++i) {
      if (elect_one()) load_s(kb0 + i, i);
      __syncwarp();
    }
    int s = 0;
    uint32_t phase = 0;              // stage s is refilled once its first contents have been consumed
    for (int kb = kb0 + pre; kb < kb1; ++kb) {
      if (!warp_all(mbar_wait(&empty[s], phase, p.status, AXB_TIMEOUT_EMPTY))) break;
      if (elect_one()) {
        mbar_expect_tx(&full[s], C::STAGE);
        load_p(kb, s);
        load_s(kb, s);
      }
      __syncwarp();
      if (++s == C::STAGES) {
        s = 0;
        phase ^= 1;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(SK_BM, NT, 0, 0);
    const uint64_t base = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
    int s = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!warp_all(mbar_wait(&full[s], phase, p.status, AXB_TIMEOUT_FULL))) break;
      tc_fence_after();
      const uint64_t a = base + (uint32_t)(s * (C::STAGE / 16)), b = a + SK_P_BYTES / 16;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < SK_BK / 16; ++kk) umma_f16(tmem, a + kk * 2, b + kk * 2, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == C::STAGES) {
        s = 0;
        phase ^= 1;
      }
    }
    if (elect_one()) umma_commit(done);
  }
  __syncwarp();
  warp_all(mbar_wait(done, 0, p.status, AXB_TIMEOUT_TMEM_FULL));
  tc_fence_after();
  pdl_wait();
  // partial tile, [n][128] fp32 in the ring (every load into it has been consumed by a retired MMA)
  float* part = reinterpret_cast<float*>(smem);
#pragma unroll 1
  for (int c = 0; c < NT / 16; ++c) {
    if (c * 16 >= p.N) break;
    uint32_t r[16];
    tmem_ld_32x16(tmem + (uint32_t(warp * 32) << 16) + c * 16, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) part[(c * 16 + j) * SK_BM + warp * 32 + lane] = __uint_as_float(r[j]);
  }
  tc_fence_before();
  if (cs > 1) cluster_sync();
  else __syncthreads();
  const uint32_t pbase = smem_u32(part);
  auto sum4 = [&](int off) {           // part[off .. off + 3], summed over the cluster in rank order
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (cs == 1) {
      a = *reinterpret_cast<const float4*>(part + off);
    } else {
#pragma unroll 4
      for (int q = 0; q < cs; ++q) {
        const float4 v = ld_cluster_f32x4(mapa_u32(pbase + off * 4, q));
        a.x += v.x;
        a.y += v.y;
        a.z += v.z;
        a.w += v.w;
      }
    }
    return a;
  };
  if (p.out_mode == 1) {
    const int n4 = (p.N + 3) / 4;
    for (int i = rank * SK_T + tid; i < n4 * SK_BM; i += cs * SK_T) {
      const int rr = i % SK_BM, n0 = (i / SK_BM) * 4;
      const long long row = (long long)tile * SK_BM + rr;
      if (row >= p.R) continue;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      for (int q = 0; q < cs; ++q)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += ld_cluster_f32(mapa_u32(pbase + ((n0 + j) * SK_BM + rr) * 4, q));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (n0 + j >= p.N) break;
        if (p.out_f32) reinterpret_cast<float*>(p.C)[row * p.ldc + n0 + j] = v[j] * p.alpha;
        else reinterpret_cast<__nv_bfloat16*>(p.C)[row * p.ldc + n0 + j] = __float2bfloat16(v[j] * p.alpha);
      }
    }
  } else {
    const int q4 = glu ? 16 : 32;      // groups of four consecutive r in a tile
    const bool vec = (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.C) & (p.out_f32 ? 15 : 7)) == 0;
    for (int i = rank * SK_T + tid; i < p.N * q4; i += cs * SK_T) {
      const int n = i / q4, rr = (i % q4) * 4;
      const int r0 = tile * (glu ? 64 : SK_BM) + rr;
      if (r0 >= p.R) continue;
      const float4 a = sum4(n * SK_BM + rr);
      float v[4] = {a.x * p.alpha, a.y * p.alpha, a.z * p.alpha, a.w * p.alpha};
      if (glu) {
        const float4 b = sum4(n * SK_BM + 64 + rr);
        const float u[4] = {b.x * p.alpha, b.y * p.alpha, b.z * p.alpha, b.w * p.alpha};
        const float L = p.glu_limit;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float gc = L > 0.f ? fminf(v[j], L) : v[j];
          const float uc = L > 0.f ? fminf(fmaxf(u[j], -L), L) : u[j];
          v[j] = sk_act(gc, p.glu_kind) * uc;
        }
      } else if (p.bias) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (r0 + j < p.R) v[j] += __bfloat162float(p.bias[r0 + j]);
      }
      if (p.out_f32) {
        float* c = reinterpret_cast<float*>(p.C) + (long long)n * p.ldc + r0;
        if (vec && r0 + 4 <= p.R) *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
        else
          for (int j = 0; j < 4 && r0 + j < p.R; ++j) c[j] = v[j];
      } else {
        __nv_bfloat16* c = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)n * p.ldc + r0;
        if (vec && r0 + 4 <= p.R) *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
        else
          for (int j = 0; j < 4 && r0 + j < p.R; ++j) c[j] = __float2bfloat16(v[j]);
      }
    }
  }
  if (cs > 1) cluster_sync();          // peers may still read this CTA's partial tile
  else __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

template <int NT>
int launch_skinny(const CUtensorMap& tP, const CUtensorMap& tS, const CUtensorMap& tP2, const CUtensorMap& tS2,
                  const SkinnyParams& p, int tiles, int splits, bool pdl, cudaStream_t st) {
  using C = SkCfg<NT>;
  auto kern = gemm_skinny_kernel<NT>;
  static std::atomic<unsigned long long> allowed{0};
  if (const int rc = axb_allow_smem((const void*)kern, C::SMEM, allowed)) return rc;
  AxbLaunch l(dim3((unsigned)(tiles * splits)), SK_T, C::SMEM, st, splits, pdl);
  const cudaError_t e = cudaLaunchKernelEx(&l.cfg, kern, tP, tS, tP2, tS2, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// CTAs per tile: the largest cluster of which the chip holds one per tile at once, at least two K blocks for each CTA. Two CTAs
// share an SM but a cluster stays inside one GPC, so that 33 clusters of eight are resident, 70 of four, 92 of three and 148 of
// two; one more is a second wave (seen as the step in time against the number of tiles; the runtime's occupancy query counts
// one CTA per SM for clusters). 48 columns, K = 4096: 33 / 35 tiles take 21.5 / 29.5 us with eight CTAs each and 23.5 with
// four, 74 tiles 37.9 with four and 31.7 with three, 96 tiles 46.1 with three and 37.9 with two. Clusters of 5 to 7 pack
// badly (6144 x 4096, 8 tokens: 20.5 us with 4, 26.6 us with 6, 24.6 us with 8 CTAs per tile).
int pick_splits(int tiles, int nk) {
  const int sizes[][2] = {{8, 33}, {4, 70}, {3, 92}, {2, 148}};
  for (const auto& s : sizes)
    if (tiles <= s[1] && nk >= 2 * s[0]) return s[0];
  return 1;
}

}  // namespace

// See the head of this file. P [R, K] (out_mode 2: [2R, K]), S [N, K], P2 / S2 the K-extension (K2 = 0: none); rows of all four
// are 16-byte aligned with strides that are multiples of 8 elements. p_dep: P, too, is written by the launch before this one.
// splits: 0 = chosen by pick_splits. pdl: the launch may overlap the end of its predecessor.
extern "C" int axb_gemm_skinny(const void* P, long long ldp, const void* S, long long lds, void* C, long long ldc, int R, int N,
                               int K, const void* P2, long long ldp2, const void* S2, long long lds2, int K2, float alpha,
                               const void* bias, int out_mode, int out_f32, int glu_kind, float glu_limit, int p_dep, int splits,
                               int pdl, int* status, void* stream) {
  if (R <= 0 || N <= 0 || (K <= 0 && K2 <= 0)) return 0;
  if (N > 256 || out_mode < 0 || out_mode > 2 || splits < 0 || splits > 8) return -2;
  if (out_mode == 2 && (out_f32 || (R % 64) || glu_kind < 0 || glu_kind > 1)) return -2;
  if (K <= 0) return -2;
  if (N > 128) {
    const long long c_off = 128ll * (out_mode == 1 ? 1 : ldc) * (out_f32 ? 4 : 2);
    const int rc = axb_gemm_skinny(P, ldp, S, lds, C, ldc, R, 128, K, P2, ldp2, S2, lds2, K2, alpha, bias, out_mode, out_f32, glu_kind,
                                   glu_limit, p_dep, splits, pdl, status, stream);
    return rc ? rc : axb_gemm_skinny(P, ldp, (const __nv_bfloat16*)S + 128 * lds, lds, (uint8_t*)C + c_off, ldc, R, N - 128, K, P2, ldp2,
                                     K2 > 0 ? (const __nv_bfloat16*)S2 + 128 * lds2 : nullptr, lds2, K2, alpha, bias, out_mode, out_f32,
                                     glu_kind, glu_limit, p_dep, splits, pdl, status, stream);
  }
  const int NT = N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : 128));
  const int prow = out_mode == 2 ? 64 : SK_BM;
  const uint64_t rows = (uint64_t)R * (out_mode == 2 ? 2 : 1);
  CUtensorMap tP, tS, tP2, tS2;
  int rc = axb_make_tmap_2d(&tP, P, rows, K, ldp, prow, SK_BK);
  if (!rc) rc = axb_make_tmap_2d(&tS, S, N, K, lds, NT, SK_BK);
  tP2 = tP;
  tS2 = tS;
  if (!rc && K2 > 0) {
    rc = axb_make_tmap_2d(&tP2, P2, rows, K2, ldp2, prow, SK_BK);
    if (!rc) rc = axb_make_tmap_2d(&tS2, S2, N, K2, lds2, NT, SK_BK);
  }
  if (rc) return -100 - rc;
  SkinnyParams p;
  p.C = C;
  p.ldc = ldc;
  p.bias = (const __nv_bfloat16*)bias;
  p.R = R;
  p.N = N;
  p.K = K;
  p.K2 = K2 > 0 ? K2 : 0;
  p.alpha = alpha;
  p.out_mode = out_mode;
  p.out_f32 = out_f32;
  p.p_dep = p_dep;
  p.glu_kind = glu_kind;
  p.glu_limit = glu_limit;
  p.status = status;
  const int tiles = (R + prow - 1) / prow;
  const int nk = (K + SK_BK - 1) / SK_BK + (p.K2 + SK_BK - 1) / SK_BK;
  if (splits == 0) splits = pick_splits(tiles, nk);
  if (splits > nk) splits = nk;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (NT) {
    case 16: return launch_skinny<16>(tP, tS, tP2, tS2, p, tiles, splits, pdl != 0, st);
    case 32: return launch_skinny<32>(tP, tS, tP2, tS2, p, tiles, splits, pdl != 0, st);
    case 64: return launch_skinny<64>(tP, tS, tP2, tS2, p, tiles, splits, pdl != 0, st);
    default: return launch_skinny<128>(tP, tS, tP2, tS2, p, tiles, splits, pdl != 0, st);
  }
}
