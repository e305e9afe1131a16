// Grouped expert GEMM with NVFP4 weights decoded inside the kernel (W4A16): the bf16 weight stack of a
// mixture-of-experts projection never exists in global memory.
//
//   FWD  C[rows, N] = alpha * (A[rows, K] . W[e]^T + A2[rows, K2] . W2[e]^T)     W[e] logical [N, K]
//   DX   C[rows, K] = alpha * (A[rows, N] . W[e]   + A2[rows, K2] . W2[e])       (input gradient)
//
// W is stored as packed E2M1 nibbles [E, N, K/2] (low nibble = even k), E4M3 block scales [E, N, K/16] and
// one fp32 scale per expert; W2 / A2 (the LoRA K-extension) are bf16. Rows are expert-sorted and padded to
// 128-row blocks (blk_expert[b] = expert of block b), exactly as in grouped_gemm.cu.
//
// Per k block TMA brings the bf16 A tiles and the PACKED weight tile (4 KB instead of 16 KB)
// into shared memory; converter warps expand the nibbles and write the bf16 tile in the
// 128-byte-swizzled layout tcgen05.mma reads; the MMA warp accumulates in TMEM; four epilogue warps store
// the result. One decoded weight tile feeds TWO 128-row blocks of the same expert (256 rows per pass), which
// halves the decode work per FLOP. The decode builds, per 16-value scale group, the eight products
// |e2m1| x scale as bf16 (one fp32 multiply for 1.5 x scale; the power-of-two multiples are exponent
// offsets of the same two roundings) and picks them with byte permutes, about 2.6 instructions per value.
// The decoded values are bit-identical to nvfp4_dequant_kernel's, so the product equals
// dequantise-then-GEMM exactly, at a quarter of the weight traffic and without the bf16 scratch. This is the role the Marlin W4A16 grouped kernel and the
// dequantise-into-a-chunk path play in the reference
// (src/axolotl/integrations/kernels/libs/scattermoe_lora/marlin_w4a16/_csrc/libtorch_stable/moe/marlin_moe_wna16/marlin_template.h:251,
//  src/axolotl/integrations/kernels/libs/scattermoe_lora/grouped_train.py:446-596).
#include "axb_common.cuh"

namespace {

constexpr int BM = 128;
constexpr int BN = 128;
constexpr int BK = 64;
constexpr int W4_CONV_WARPS = 16;
constexpr int W4_THREADS = 192 + 32 * W4_CONV_WARPS + 32;   // TMA (A), MMA, 4 epilogue warps, converters, TMA (weights)
// Three rings of their own: the packed weights are small and run four k blocks ahead of the decode;
// a slot of the decoded tile is only held from its decode to its MMA, and a slot of A from its load to its MMA.
// The converters work in four groups of four warps, each on a k block of its own, so that four chains (packed tile seen ->
// decode -> stores -> proxy fence -> arrival) run side by side. Two warps a group left the decode's dependent instructions
// uncovered: 512 rows of each of 128 experts, 2048 -> 1536 393 -> 366 us, 768 -> 2048 220 -> 199.
constexpr int SA = 4, SB = 4, SR = 4;  // slots: A (two 128-row tiles), decoded B, packed B
// Every group owns one slot of the packed and one of the decoded ring (k block i of the whole sequence belongs to group, slot
// i % 4), so that a slot's waits are made in order by the same warps: a wait for a phase whose predecessor has not completed
// would see the parity it asks for and pass.
constexpr int CGROUPS = 4, CG_WARPS = W4_CONV_WARPS / CGROUPS, CG_UNITS = 256 / (32 * CG_WARPS);
constexpr int A_BYTES = BM * BK * 2;   // one 128-row A tile; a slot holds two
constexpr int B_BYTES = BN * BK * 2;
constexpr int RAW_BYTES = 4096;   // FWD: 128 rows x 32 bytes; DX: 64 rows x 64 bytes
constexpr int EPI_BYTES = 4096;   // per epilogue warp: 32 rows x 64 bf16 columns on their way out
constexpr int W4_SMEM = SA * 2 * A_BYTES + SB * B_BYTES + SR * RAW_BYTES + 4 * EPI_BYTES + 1024 + 512;
static_assert(W4_SMEM <= 227 * 1024 && SB == CGROUPS && SR % CGROUPS == 0, "");

constexpr int PF = 8;                  // k blocks between a packed tile's L2 prefetch and its load
AXB_DEVICE void tma_prefetch_3d(const CUtensorMap* tmap, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0),
               "r"(c1), "r"(c2)
               : "memory");
}
// position in a ring of N slots
template <int N>
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  AXB_DEVICE void next() {
    if (++slot == N) {
      slot = 0;
      phase ^= 1;
    }
  }
};

// E4M3 byte -> fp32, branch free: the 7 magnitude bits placed at the top of an fp32 mantissa / the bottom of
// its exponent give value x 2^-120 (subnormal inputs included), and 0x7F / 0xFF are NaN. Same value as
// the table-free decode of nvfp4_dequant_kernel.
AXB_DEVICE float e4m3_to_float(uint32_t v) {
  const uint32_t mag = v & 0x7Fu;
  float f = __uint_as_float(mag << 20) * 1.329227995784916e36f;   // 2^120
  f = mag == 0x7Fu ? __int_as_float(0x7fc00000) : f;
  return __uint_as_float(__float_as_uint(f) | ((v & 0x80u) << 24));
}
AXB_DEVICE uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// The eight bf16 products |code| x s of one scale group, split into low-byte and high-byte tables for prmt.
// |code| = 0, .5, 1, 1.5, 2, 3, 4, 6: bf16(fp32(m x s)) for m a power of two is bf16(s) with the exponent
// moved, and 3 s, 6 s are 1.5 s with the exponent moved, so two roundings give all eight (same bits as
// rounding each fp32 product) as long as no exponent leaves the normal range; otherwise multiply them out.
struct Lut {
  uint32_t L0, L1, H0, H1;
};
AXB_DEVICE Lut make_lut(float s) {
  const uint32_t P23 = pack_bf16x2(s, 1.5f * s);   // low half: 1 x s, high half: 1.5 x s
  uint32_t P01, P45, P67;
  if (((P23 >> 7) & 0x1FFu) - 2u < 0xFAu) {        // s positive, exponent in [2, 251]
    P01 = (P23 << 16) - 0x00800000u;               // (0, 0.5 s)
    P45 = P23 + 0x00800080u;                       // (2 s, 3 s)
    P67 = P23 + 0x01000100u;                       // (4 s, 6 s)
  } else {
    P01 = pack_bf16x2(0.f * s, 0.5f * s);
    P45 = pack_bf16x2(2.f * s, 3.f * s);
    P67 = pack_bf16x2(4.f * s, 6.f * s);
  }
  Lut t;
  t.L0 = prmt(P01, P23, 0x6420);
  t.H0 = prmt(P01, P23, 0x7531);
  t.L1 = prmt(P45, P67, 0x6420);
  t.H1 = prmt(P45, P67, 0x7531);
  return t;
}
// 8 packed codes (one 32-bit word, low nibble first) -> 8 bf16 in a 16-byte chunk
AXB_DEVICE uint4 decode8(uint32_t w, const Lut& t) {
  const uint32_t sel = w & 0x77777777u, selh = sel >> 16;
  const uint32_t sg = w & 0x88888888u, sg4 = sg << 4;   // sign of odd codes / even codes at bit 7 of byte i/2
  uint32_t lo = prmt(t.L0, t.L1, sel), hi = prmt(t.H0, t.H1, sel);
  hi ^= prmt(sg4, sg, 0x5140) & 0x80808080u;
  uint4 o;
  o.x = prmt(lo, hi, 0x5140);
  o.y = prmt(lo, hi, 0x7362);
  lo = prmt(t.L0, t.L1, selh);
  hi = prmt(t.H0, t.H1, selh);
  hi ^= prmt(sg4, sg, 0x7362) & 0x80808080u;
  o.z = prmt(lo, hi, 0x5140);
  o.w = prmt(lo, hi, 0x7362);
  return o;
}

struct W4Params {
  int N, K, K2;   // FWD: N output columns, K contraction. DX: N = output columns (the weight's K), K = contraction (the weight's N)
  int Wn, Wk;     // logical weight shape [Wn, Wk] per expert
  int E;
  void* C;
  long long ldc;
  float alpha;
  int out_mode;   // 0 bf16, 1 fp32
  int tma_store;  // bf16 rows leave through staging tiles and TMA stores (row stores of 32 lanes, a line each, held up the converters)
  const uint8_t* scale;   // [E, Wn, Wk / 16] e4m3 bytes
  const float* pts;       // [E]
  const int* blk_expert;
  const int* n_blocks;
  int* status;
};

// tensor map over the packed weight bytes [E, Wn, Wk/2], box [1, box_rows, box_bytes], no swizzle
int make_tmap_u8_3d(CUtensorMap* out, const void* base, uint64_t batch, uint64_t rows, uint64_t row_bytes,
                    uint32_t box_rows, uint32_t box_bytes) {
  AxbEncodeTiledFn fn = axb_get_encode_fn();
  if (!fn) return -1;
  cuuint64_t dims[3] = {row_bytes, rows, batch};
  cuuint64_t strides[2] = {row_bytes, rows * row_bytes};
  cuuint32_t box[3] = {box_bytes, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = CUDA_SUCCESS;
  for (int attempt = 0; attempt < 2; ++attempt) {
    r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_ERROR_INVALID_CONTEXT) break;
    cudaFree(nullptr);
  }
  return r == CUDA_SUCCESS ? 0 : (int)r;
}

// One pass = one decoded weight tile stream against one or two 128-row blocks of the same expert.
struct Pass {
  int blk, two, e, n0;
};
// Tiles are (pair of consecutive row blocks, n block). Sub-pass 0 takes block 2p (and 2p+1 when it belongs to
// the same expert); sub-pass 1 exists only when block 2p+1 belongs to another expert.
AXB_DEVICE bool get_pass(const int* blk_expert, int n_blocks, int num_n, int E, int tile, int sub, Pass& ps) {
  const int pair = tile / num_n;
  const int b0 = 2 * pair, b1 = b0 + 1;
  int e0 = blk_expert[b0];
  const bool has1 = b1 < n_blocks;
  int e1 = has1 ? blk_expert[b1] : -1;
  if (!AXB_INDEX_OK(AXB_SITE_W4A16_EXPERT, e0, E)) e0 = 0;              // checked build: recorded, then a valid expert
  if (has1 && !AXB_INDEX_OK(AXB_SITE_W4A16_EXPERT, e1, E)) e1 = 0;
  ps.n0 = (tile - pair * num_n) * BN;
  if (sub == 0) {
    ps.blk = b0;
    ps.two = has1 && e1 == e0;
    ps.e = e0;
    return true;
  }
  if (!has1 || e1 == e0) return false;
  ps.blk = b1;
  ps.two = 0;
  ps.e = e1;
  return true;
}

template <bool DX>
__global__ void __launch_bounds__(W4_THREADS, 1)
    grouped_w4a16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmQ,
                         const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2,
                         const __grid_constant__ CUtensorMap tmC, const W4Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;                                   // [slot][2][128 x 64]
  uint8_t* sB = smem + SA * 2 * A_BYTES;
  uint8_t* sRaw = sB + SB * B_BYTES;
  uint8_t* sEpi = sRaw + SR * RAW_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sEpi + 4 * EPI_BYTES);
  uint64_t* a_full = bars;                      // A tiles landed
  uint64_t* a_empty = a_full + SA;              // their MMAs retired
  uint64_t* b_full = a_empty + SA;              // bf16 B tile in place (one arrival per warp of its group; the LoRA tile by TMA)
  uint64_t* b_empty = b_full + SB;
  uint64_t* r_full = b_empty + SB;              // packed weights landed
  uint64_t* r_empty = r_full + SR;              // read by its group
  uint64_t* tfull_bar = r_empty + SR;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int n_blocks = *p.n_blocks;
  const int num_n = (p.N + BN - 1) / BN;
  const int nk_main = (p.K + BK - 1) / BK, nk_ext = (p.K2 + BK - 1) / BK;
  const int nk = nk_main + nk_ext;
  const int total = ((n_blocks + 1) / 2) * num_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < SA; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < SB; ++s) {
      mbar_init(&b_full[s], CG_WARPS);
      mbar_init(&b_empty[s], 1);
    }
    for (int s = 0; s < SR; ++s) {
      mbar_init(&r_full[s], 1);
      mbar_init(&r_empty[s], CG_WARPS);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull_bar[s], 1);
      mbar_init(&tempty_bar[s], 4);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmQ);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);   // two accumulator slots of 2 x 128 columns
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ A tiles
    Ring<SA> ra;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      for (int sub = 0; sub < 2 && ok; ++sub) {
        Pass ps;
        if (!get_pass(p.blk_expert, n_blocks, num_n, p.E, tile, sub, ps)) continue;
        const uint32_t a_bytes = ps.two ? 2 * A_BYTES : A_BYTES;
        for (int kb = 0; kb < nk; ++kb, ra.next()) {
          if (!warp_all(mbar_wait(&a_empty[ra.slot], ra.phase ^ 1, p.status, AXB_TIMEOUT_EMPTY))) {
            ok = false;
            break;
          }
          const bool ext = kb >= nk_main;
          uint8_t* a_dst = sA + ra.slot * 2 * A_BYTES;
          const CUtensorMap* ma = ext ? &tmA2 : &tmA;
          const int ka = ext ? (kb - nk_main) * BK : kb * BK;
          if (elect_one()) {
            mbar_expect_tx(&a_full[ra.slot], a_bytes);
            tma_load_2d(a_dst, ma, &a_full[ra.slot], ka, ps.blk * BM);
            if (ps.two) tma_load_2d(a_dst + A_BYTES, ma, &a_full[ra.slot], ka, (ps.blk + 1) * BM);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp == W4_THREADS / 32 - 1) {
    // ------------------------------------------------------------ packed weights
    // They come from DRAM, and four slots do not cover that latency where an expert has few rows: a second walk over the same
    // sequence asks for them PF k blocks earlier, into L2 (20 rows of each of 128 experts, 2048 -> 1536: 221 -> 190 us,
    // 768 -> 2048: 109 -> 94; 16 blocks ahead is no better; with 512 rows an expert it makes no difference). More slots would do
    // the same and cost the A ring one.
    int pt = blockIdx.x, psub = 0, pkb = 0;
    Pass pp;
    bool live = pt < total && get_pass(p.blk_expert, n_blocks, num_n, p.E, pt, 0, pp);
    auto prefetch_step = [&]() {
      if (!live) return;
      if (pkb < nk_main && elect_one()) {
        if (!DX) tma_prefetch_3d(&tmQ, pkb * (BK / 2), pp.n0, pp.e);
        else tma_prefetch_3d(&tmQ, pp.n0 / 2, pkb * BK, pp.e);
      }
      __syncwarp();
      if (++pkb < nk) return;
      pkb = 0;
      do {
        if (++psub == 2) psub = 0, pt += gridDim.x;
        live = pt < total;
      } while (live && !get_pass(p.blk_expert, n_blocks, num_n, p.E, pt, psub, pp));
    };
    for (int i = 0; i < PF; ++i) prefetch_step();
    Ring<SR> rr;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      for (int sub = 0; sub < 2 && ok; ++sub) {
        Pass ps;
        if (!get_pass(p.blk_expert, n_blocks, num_n, p.E, tile, sub, ps)) continue;
        for (int kb = 0; kb < nk; ++kb, rr.next()) {
          prefetch_step();
          if (!warp_all(mbar_wait(&r_empty[rr.slot], rr.phase ^ 1, p.status, AXB_TIMEOUT_EMPTY))) {
            ok = false;
            break;
          }
          if (kb >= nk_main) {          // a LoRA block has no packed weights: its slot only keeps the order
            if (elect_one()) mbar_arrive(&r_full[rr.slot]);
          } else if (elect_one()) {
            mbar_expect_tx(&r_full[rr.slot], RAW_BYTES);
            if (!DX) tma_load_3d(sRaw + rr.slot * RAW_BYTES, &tmQ, &r_full[rr.slot], kb * (BK / 2), ps.n0, ps.e);   // [128 n, 32 B of k]
            else tma_load_3d(sRaw + rr.slot * RAW_BYTES, &tmQ, &r_full[rr.slot], ps.n0 / 2, kb * BK, ps.e);         // [64 n, 64 B of k]
          }
          __syncwarp();
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issue
    constexpr uint32_t idesc = make_idesc_bf16(BM, BN, 0, DX ? 1 : 0);
    const uint64_t da_base = make_smem_desc_sw128(smem_u32(sA), 16, 1024);
    const uint64_t db_base = DX ? make_smem_desc_sw128(smem_u32(sB), 8192, 1024) : make_smem_desc_sw128(smem_u32(sB), 16, 1024);
    Ring<SA> ra;
    Ring<SB> rb;
    int it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      for (int sub = 0; sub < 2 && ok; ++sub) {
        Pass ps;
        if (!get_pass(p.blk_expert, n_blocks, num_n, p.E, tile, sub, ps)) continue;
        const int acc = it & 1;
        if (!warp_all(mbar_wait(&tempty_bar[acc], ((it >> 1) & 1) ^ 1, p.status, AXB_TIMEOUT_TMEM_EMPTY))) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 2 * BN;
        for (int kb = 0; kb < nk; ++kb, ra.next(), rb.next()) {
          if (!warp_all(mbar_wait(&a_full[ra.slot], ra.phase, p.status, AXB_TIMEOUT_FULL) &&
                        mbar_wait(&b_full[rb.slot], rb.phase, p.status, AXB_TIMEOUT_FULL))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t da = da_base + (uint32_t)(ra.slot * (2 * A_BYTES / 16)), db = db_base + (uint32_t)(rb.slot * (B_BYTES / 16));
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              const uint64_t dbk = db + kk * (DX ? 2048 / 16 : 32 / 16);
              const uint32_t accum = (kb > 0 || kk > 0) ? 1u : 0u;
              umma_f16(d_tmem, da + kk * 2, dbk, idesc, accum);
              if (ps.two) umma_f16(d_tmem + BN, da + A_BYTES / 16 + kk * 2, dbk, idesc, accum);
            }
            umma_commit(&a_empty[ra.slot]);
            umma_commit(&b_empty[rb.slot]);
            if (kb == nk - 1) umma_commit(&tfull_bar[acc]);
          }
          __syncwarp();
        }
        ++it;
      }
    }
  } else if (warp >= 6) {
    // ------------------------------------------------------------ converters: packed tile -> bf16 B tile
    // A k block is 256 units of 16 packed bytes (32 codes, 2 scale groups); thread t of a group takes units t, t + 128
    // Unit ct lies at raw + ct * 16 and becomes four 16-byte chunks of the swizzled bf16 tile.
    //   FWD: raw tile [128 n][32 B]: weight row n0 + ct / 2, codes 32 * (ct & 1) .. + 31 of k block kb
    //        -> K-major row ct / 2, chunks 4 * (ct & 1) .. + 3.
    //   DX : raw tile [64 wn][64 B]: weight row kb * 64 + ct / 4, columns n0 + 64 * half + 32 * part .. + 31
    //        (half = (ct >> 1) & 1, part = ct & 1) -> MN-major chunk block `half`, row ct / 4, chunks 4 * part .. + 3.
    // Shared-memory accesses are conflict free: the loads are contiguous, and the eight lanes of a store phase
    // hit eight different 16-byte chunk positions (rows differ in swizzle bits 0-1 or bit 0, `part` flips bit 2,
    // and in dX the odd half walks its chunks in the order 2, 3, 0, 1, which flips bit 1).
    const int cw = warp - 6, grp = cw / CG_WARPS, gt = (cw % CG_WARPS) * 32 + lane;
    const long long sc_row_bytes = p.Wk / 16;
    const int part = gt & 1, half = DX ? ((gt >> 1) & 1) : 0;      // the same for all units of a thread
    long long cb = 0;                                             // k blocks before this pass
    bool ok = true;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      for (int sub = 0; sub < 2 && ok; ++sub) {
        Pass ps;
        if (!get_pass(p.blk_expert, n_blocks, num_n, p.E, tile, sub, ps)) continue;
        const float g = p.pts[ps.e];
        const uint8_t* sc_base = p.scale + (long long)ps.e * p.Wn * sc_row_bytes;
        // the two E4M3 bytes of each unit, requested one turn (four k blocks) ahead and looked at when they are needed
        auto load_scales = [&](int kb, uint32_t (&out)[CG_UNITS]) {
#pragma unroll
          for (int u = 0; u < CG_UNITS; ++u) {
            out[u] = 0u;
            const int ct = gt + u * (256 / CG_UNITS);
            if (kb >= nk_main) continue;
            if (!DX) {
              const int n = ps.n0 + (ct >> 1);
              if (n < p.Wn) out[u] = __ldg(reinterpret_cast<const unsigned short*>(sc_base + (long long)n * sc_row_bytes + kb * 4 + part * 2));
            } else {
              const int k0 = ps.n0 + half * 64 + part * 32, wn = kb * BK + (ct >> 2);
              if (k0 < p.Wk && wn < p.Wn)
                out[u] = __ldg(reinterpret_cast<const unsigned short*>(sc_base + (long long)wn * sc_row_bytes + k0 / 16));
            }
          }
        };
        // this group's k blocks of the pass: every fourth of the whole sequence
        int kb = (int)((grp - cb) & (CGROUPS - 1));
        uint32_t cur[CG_UNITS], nxt[CG_UNITS];
        load_scales(kb, cur);
        for (; kb < nk && ok; kb += CGROUPS) {
          load_scales(kb + CGROUPS, nxt);
          const int bslot = grp, rslot = (int)((cb + kb) % SR);
          const uint32_t bphase = (uint32_t)((cb + kb) / SB) & 1, rphase = (uint32_t)((cb + kb) / SR) & 1;
          if (!mbar_wait(&r_full[rslot], rphase, p.status, AXB_TIMEOUT_FULL)) {
            ok = false;
            break;
          }
          if (kb < nk_main) {
            uint4 w[CG_UNITS];
#pragma unroll
            for (int u = 0; u < CG_UNITS; ++u)
              w[u] = *reinterpret_cast<const uint4*>(sRaw + rslot * RAW_BYTES + (gt + u * (256 / CG_UNITS)) * 16);
            if (!mbar_wait(&b_empty[bslot], bphase ^ 1, p.status, AXB_TIMEOUT_EMPTY)) {
              ok = false;
              break;
            }
#pragma unroll
            for (int u = 0; u < CG_UNITS; ++u) {
              const int ct = gt + u * (256 / CG_UNITS), r = DX ? (ct >> 2) : (ct >> 1);
              uint32_t sc2 = cur[u];
              int pos = (part * 4) ^ (r & 7);           // chunk position of this unit's first chunk
              if (DX && half) {
                w[u] = make_uint4(w[u].z, w[u].w, w[u].x, w[u].y);
                sc2 = ((sc2 >> 8) | (sc2 << 8)) & 0xFFFFu;
                pos ^= 2;
              }
              uint8_t* dst_row = sB + bslot * B_BYTES + half * 8192 + r * 128;
              Lut t = make_lut(e4m3_to_float(sc2 & 0xFF) * g);
              *reinterpret_cast<uint4*>(dst_row + ((pos ^ 0) << 4)) = decode8(w[u].x, t);
              *reinterpret_cast<uint4*>(dst_row + ((pos ^ 1) << 4)) = decode8(w[u].y, t);
              t = make_lut(e4m3_to_float(sc2 >> 8) * g);
              *reinterpret_cast<uint4*>(dst_row + ((pos ^ 2) << 4)) = decode8(w[u].z, t);
              *reinterpret_cast<uint4*>(dst_row + ((pos ^ 3) << 4)) = decode8(w[u].w, t);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(&b_full[bslot]);
              mbar_arrive(&r_empty[rslot]);
            }
          } else {                                    // the LoRA tile comes by TMA, on the group's first arrival
            if (!mbar_wait(&b_empty[bslot], bphase ^ 1, p.status, AXB_TIMEOUT_EMPTY)) {
              ok = false;
              break;
            }
            if (lane == 0) {
              mbar_arrive(&r_empty[rslot]);
              if (cw % CG_WARPS == 0) {
                const int ka = (kb - nk_main) * BK;
                uint8_t* b_dst = sB + bslot * B_BYTES;
                mbar_expect_tx(&b_full[bslot], B_BYTES);
                if (!DX) {
                  tma_load_3d(b_dst, &tmB2, &b_full[bslot], ka, ps.n0, ps.e);
                } else {
                  tma_load_3d(b_dst, &tmB2, &b_full[bslot], ps.n0, ka, ps.e);
                  tma_load_3d(b_dst + 8192, &tmB2, &b_full[bslot], ps.n0 + 64, ka, ps.e);
                }
              } else {
                mbar_arrive(&b_full[bslot]);
              }
            }
            __syncwarp();
          }
#pragma unroll
          for (int u = 0; u < CG_UNITS; ++u) cur[u] = nxt[u];
        }
        cb += nk;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps 2..5
    const int lane_group = warp & 3;
    int it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
      for (int sub = 0; sub < 2 && ok; ++sub) {
        Pass ps;
        if (!get_pass(p.blk_expert, n_blocks, num_n, p.E, tile, sub, ps)) continue;
        const int acc = it & 1;
        if (!mbar_wait(&tfull_bar[acc], (it >> 1) & 1, p.status, AXB_TIMEOUT_TMEM_FULL)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int h = 0; h <= ps.two; ++h) {
          if (p.tma_store) {
            const uint32_t t_row = tmem_base + (uint32_t(lane_group * 32) << 16) + acc * 2 * BN + h * BN;
            uint8_t* tile_out = sEpi + lane_group * EPI_BYTES;
#pragma unroll 1
            for (int c = 0; c < BN / 64; ++c) {
              if (ps.n0 + c * 64 >= p.N) break;
              uint32_t r[2][32];
              tmem_ld_32x32(t_row + c * 64, r[0]);
              tmem_ld_32x32(t_row + c * 64 + 32, r[1]);
              tmem_ld_wait();
              uint4 w[8];
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const uint32_t* v = &r[q >> 2][(q & 3) * 8];
                w[q] = make_uint4(pack_bf16x2(__uint_as_float(v[0]) * p.alpha, __uint_as_float(v[1]) * p.alpha),
                                  pack_bf16x2(__uint_as_float(v[2]) * p.alpha, __uint_as_float(v[3]) * p.alpha),
                                  pack_bf16x2(__uint_as_float(v[4]) * p.alpha, __uint_as_float(v[5]) * p.alpha),
                                  pack_bf16x2(__uint_as_float(v[6]) * p.alpha, __uint_as_float(v[7]) * p.alpha));
              }
              if (lane == 0) bulk_wait_group_read<0>();
              __syncwarp();
              stage_row128(tile_out, lane, w);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_store_2d(&tmC, tile_out, ps.n0 + c * 64, (ps.blk + h) * BM + lane_group * 32);
                bulk_commit_group();
              }
            }
            continue;
          }
          const long long row = (long long)(ps.blk + h) * BM + lane_group * 32 + lane;
          const uint32_t t_addr = tmem_base + (uint32_t(lane_group * 32) << 16) + acc * 2 * BN + h * BN;
#pragma unroll 1
          for (int c = 0; c < BN / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(t_addr + c * 32, r);
            tmem_ld_wait();
            const int col0 = ps.n0 + c * 32;
            if (col0 >= p.N) continue;
            const bool full_chunk = col0 + 32 <= p.N;
            if (p.out_mode == 0) {
              __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col0;
              if (full_chunk && (p.ldc & 7) == 0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  uint4 o;
                  o.x = pack_bf16x2(__uint_as_float(r[q * 8 + 0]) * p.alpha, __uint_as_float(r[q * 8 + 1]) * p.alpha);
                  o.y = pack_bf16x2(__uint_as_float(r[q * 8 + 2]) * p.alpha, __uint_as_float(r[q * 8 + 3]) * p.alpha);
                  o.z = pack_bf16x2(__uint_as_float(r[q * 8 + 4]) * p.alpha, __uint_as_float(r[q * 8 + 5]) * p.alpha);
                  o.w = pack_bf16x2(__uint_as_float(r[q * 8 + 6]) * p.alpha, __uint_as_float(r[q * 8 + 7]) * p.alpha);
                  *reinterpret_cast<uint4*>(crow + q * 8) = o;
                }
              } else {
                for (int j = 0; j < 32 && col0 + j < p.N; ++j) crow[j] = __float2bfloat16(__uint_as_float(r[j]) * p.alpha);
              }
            } else {
              float* crow = reinterpret_cast<float*>(p.C) + row * p.ldc + col0;
              for (int j = 0; j < 32 && col0 + j < p.N; ++j) crow[j] = __uint_as_float(r[j]) * p.alpha;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[acc]);
        ++it;
      }
    }
    if (lane == 0) bulk_wait_group<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// A [max_blocks * 128, Ka] bf16 (lda); qdata [E, Wn, Wk/2] uint8, scale [E, Wn, Wk/16] e4m3 bytes, pts [E] fp32.
//   trans_w = 0 (forward):        Ka = Wk, C [rows, Wn];  A2 [rows, K2], W2 [E, Wn, K2] (bf16, optional)
//   trans_w = 1 (input gradient): Ka = Wn, C [rows, Wk];  A2 [rows, K2], W2 [E, K2, Wk] (bf16, optional)
// Wk must be a multiple of 64, Wn a multiple of 8; out_mode 0 bf16 / 1 fp32.
extern "C" int axb_grouped_gemm_w4a16(const void* A, long long lda, const void* qdata, const void* scale, const float* pts,
                                      const void* A2, long long lda2, const void* W2, void* C, long long ldc, int E,
                                      int Wn, int Wk, int K2, int trans_w, float alpha, int out_mode,
                                      const int* blk_expert, const int* n_blocks, int max_blocks, int* status,
                                      void* stream) {
  if (max_blocks <= 0 || Wn <= 0 || Wk <= 0) return 0;
  if ((lda & 7) || (Wk & 63) || (Wn & 7) || (K2 > 0 && ((lda2 & 7) || (K2 & 7))) || out_mode < 0 || out_mode > 1) return -2;
  const unsigned long long rows = (unsigned long long)max_blocks * BM;
  const int Ka = trans_w ? Wn : Wk, N = trans_w ? Wk : Wn;
  CUtensorMap tA, tQ, tA2, tB2, tC;
  int rc = axb_make_tmap_2d(&tA, A, rows, Ka, lda, BM, 64);
  rc |= trans_w ? make_tmap_u8_3d(&tQ, qdata, E, Wn, Wk / 2, 64, 64) : make_tmap_u8_3d(&tQ, qdata, E, Wn, Wk / 2, 128, 32);
  if (K2 > 0) {
    rc |= axb_make_tmap_2d(&tA2, A2, rows, K2, lda2, BM, 64);
    rc |= trans_w ? axb_make_tmap_3d(&tB2, W2, E, K2, Wk, Wk, (unsigned long long)Wk * K2, 64, 64)
                  : axb_make_tmap_3d(&tB2, W2, E, Wn, K2, K2, (unsigned long long)Wn * K2, BN, 64);
  } else {
    tA2 = tA;
    tB2 = tA;
  }
  const bool tma_store = out_mode == 0 && (ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  tC = tA;
  if (tma_store) rc |= axb_make_tmap_2d(&tC, C, rows, N, ldc, 32, 64);
  if (rc) return -4;
  W4Params p = {};
  p.tma_store = tma_store;
  p.N = N; p.K = Ka; p.K2 = K2 > 0 ? K2 : 0; p.Wn = Wn; p.Wk = Wk; p.E = E;
  p.C = C; p.ldc = ldc; p.alpha = alpha; p.out_mode = out_mode;
  p.scale = reinterpret_cast<const uint8_t*>(scale); p.pts = pts;
  p.blk_expert = blk_expert; p.n_blocks = n_blocks; p.status = status;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int max_tiles = ((max_blocks + 1) / 2) * ((N + BN - 1) / BN);
  int grid = sms < max_tiles ? sms : max_tiles;
  if (grid < 1) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (trans_w) {
    static bool set = false;
    if (!set) {
      cudaError_t e = cudaFuncSetAttribute(grouped_w4a16_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, W4_SMEM);
      if (e != cudaSuccess) return (int)e;
      set = true;
    }
    grouped_w4a16_kernel<true><<<grid, W4_THREADS, W4_SMEM, st>>>(tA, tQ, tA2, tB2, tC, p);
  } else {
    static bool set = false;
    if (!set) {
      cudaError_t e = cudaFuncSetAttribute(grouped_w4a16_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, W4_SMEM);
      if (e != cudaSuccess) return (int)e;
      set = true;
    }
    grouped_w4a16_kernel<false><<<grid, W4_THREADS, W4_SMEM, st>>>(tA, tQ, tA2, tB2, tC, p);
  }
  return (int)cudaGetLastError();
}
