// Grouped expert GEMM with NVFP4 weights decoded inside the kernel (W4A16): the bf16 weight stack of a
// mixture-of-experts projection never exists in global memory.
//
//   FWD  C[rows, N] = alpha * (A[rows, K] . W[e]^T + A2[rows, K2] . W2[e]^T)     W[e] logical [N, K]
//   DX   C[rows, K] = alpha * (A[rows, N] . W[e]   + A2[rows, K2] . W2[e])       (input gradient)
//
// W is stored as packed E2M1 nibbles [E, N, K/2] (low nibble = even k), E4M3 block scales [E, N, K/16] and
// one fp32 scale per expert; W2 / A2 (the LoRA K-extension) are bf16. Rows are expert-sorted and padded to
// 128-row blocks, exactly as in grouped_gemm.cu; a table lists the passes: up to two consecutive blocks of one expert.
//
// A CTA pair works on 256 weight columns x up to 256 rows. The weights are the M operand (128 columns per CTA) and the rows the N
// operand, so that a pass costs MMA time for the rows it has, to 32: an expert with 20 rows does not pay for 256. Per k block TMA
// brings half of the rows and the PACKED weight tile (4 KB instead of 16 KB) into each CTA's shared memory; converter warps expand
// the nibbles and write the bf16 tile in the 128-byte-swizzled layout tcgen05.mma reads; rank 0's MMA warp accumulates in the TMEM of
// both; four epilogue warps transpose and store. The decode picks the eight products |e2m1| x scale of a 16-value scale group, as
// bf16, with byte permutes, about 2 instructions per value; the products come from a table per expert.
// What bounds it: one CTA per 128 columns read every tile from shared memory for two MMAs (960 of 1020 clocks of a k block); the pair
// reads each half once (576). Then the chain of a k block (packed tile seen -> decode -> arrival -> MMA -> slot free), and the decode
// itself at half rate in the integer pipe: 3.1 (forward) and 3.7 (input gradient) instructions a value with table reads, addresses and
// polls, 400 and 470 of the 740 and 760 clocks that a k block takes. 128 experts with the rows of a skewed router, forward / input
// gradient, one CTA a tile -> pairs (arrivals at cluster scope included, 2 to 3 % of it), cold L2:
//   8192 x 8 rows, 2048 -> 1536  492 / 488 -> 389 / 404 us, 768 -> 2048  257 / 275 -> 245 / 199 us
//    333 x 8 rows, 2048 -> 1536  169 / 157 -> 150 / 151 us, 768 -> 2048   84 /  94 ->  87 /  89 us
//   32 experts, 2000 x 4 rows, 1024 -> 1024  40 / 42 -> 36 / 36 us
// An L2 prefetch ahead of the packed loads cost 5 % with the twelve-slot ring (it had paid with four); five or six converter groups,
// eight decoded slots and deeper packed rings changed nothing.
// The decoded values are bit-identical to nvfp4_dequant_kernel's, so the product equals
// dequantise-then-GEMM exactly, at a quarter of the weight traffic and without the bf16 scratch. This is the role the Marlin W4A16 grouped kernel and the
// dequantise-into-a-chunk path play in the reference
// (src/axolotl/integrations/kernels/libs/scattermoe_lora/marlin_w4a16/_csrc/libtorch_stable/moe/marlin_moe_wna16/marlin_template.h:251,
//  src/axolotl/integrations/kernels/libs/scattermoe_lora/grouped_train.py:446-596).
#include "axb_common.cuh"

namespace {

constexpr int BN = 256;   // weight columns of a tile, 128 per CTA
constexpr int BK = 64;
constexpr int W4_CONV_WARPS = 16;
constexpr int W4_THREADS = 192 + 32 * W4_CONV_WARPS + 32;   // TMA (rows), MMA, 4 epilogue warps, converters, TMA (packed weights)
// Three rings of their own: a slot of the decoded tile is only held from its decode to its MMA, a slot of rows from its load to
// its MMA, and the packed weights are small and run twelve k blocks ahead of the decode.
// The converters work in four groups of four warps, each on a k block of its own, so that four chains (packed tile seen ->
// decode -> stores -> proxy fence -> arrival) run side by side. Two warps a group left the decode's dependent instructions
// uncovered: 512 rows of each of 128 experts, 2048 -> 1536 393 -> 366 us, 768 -> 2048 220 -> 199 (measured when one CTA had a tile; six
// groups changed nothing in the present form).
constexpr int SX = 5, SW = 4, SR = 12;  // slots: rows, decoded weights, packed weights
// Every group owns one slot of the decoded ring and three of the packed one (k block i of the whole sequence belongs to group
// i % 4), so that a slot's waits are made in order by the same warps: a wait for a phase whose predecessor has not completed
// would see the parity it asks for and pass.
constexpr int CGROUPS = 4, CG_WARPS = W4_CONV_WARPS / CGROUPS, CG_UNITS = 256 / (32 * CG_WARPS);
constexpr int X_BYTES = 128 * BK * 2;  // this CTA's half of the rows
constexpr int W_BYTES = 128 * BK * 2;  // this CTA's half of the weight columns
constexpr int RAW_BYTES = 4096;        // FWD: 128 rows x 32 bytes; DX: 64 rows x 64 bytes
constexpr int EPI_BYTES = 4096;        // per epilogue warp: two slots of 32 rows x 32 bf16 columns on their way out
constexpr int TAB_BYTES = 128 * 16;    // per converter group: the products of every scale magnitude of its expert
constexpr int W4_SMEM = SX * X_BYTES + SW * W_BYTES + SR * RAW_BYTES + 4 * EPI_BYTES + CGROUPS * TAB_BYTES + 1024 + 512;
static_assert(W4_SMEM <= 227 * 1024 && SW % CGROUPS == 0 && SR % CGROUPS == 0 && (2 * (SX + SW + SR) + 4) * 8 + 4 <= 512, "");

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

// A wait that does not stand in the chain leaves the issue slots to the converters.
AXB_DEVICE bool wait_sleeping(uint64_t* bar, uint32_t parity, unsigned ns, int* status, int code) {
  if (mbar_test_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  uint32_t spins = 0;
  while (!mbar_test_wait(bar, parity)) {
    __nanosleep(ns);
    if ((++spins & 0xFF) == 0 && global_timer_ns() - t0 > AXB_WAIT_BUDGET_NS) {
      if (status) atomicCAS(status, 0, code);
      return false;
    }
  }
  return true;
}

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
AXB_DEVICE uint4 make_lut(float s) {
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
  // low bytes of the products of codes 0-3 and 4-7, then their high bytes
  return make_uint4(prmt(P01, P23, 0x6420), prmt(P45, P67, 0x6420), prmt(P01, P23, 0x7531), prmt(P45, P67, 0x7531));
}
// 8 packed codes (one 32-bit word, low nibble first) -> 8 bf16 in a 16-byte chunk, with the products t of make_lut
AXB_DEVICE uint4 decode8(uint32_t w, const uint4& t) {
  const uint32_t sel = w & 0x77777777u, selh = sel >> 16, w4 = w << 4;   // signs of odd (w) and even (w4) codes: bit 7 of byte i / 2
  uint32_t lo = prmt(t.x, t.y, sel), hi = prmt(t.z, t.w, sel);
  hi ^= prmt(w4, w, 0x5140) & 0x80808080u;
  uint4 o;
  o.x = prmt(lo, hi, 0x5140);
  o.y = prmt(lo, hi, 0x7362);
  lo = prmt(t.x, t.y, selh);
  hi = prmt(t.z, t.w, selh);
  hi ^= prmt(w4, w, 0x7362) & 0x80808080u;
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
  int tma_store;  // bf16 rows leave through staging tiles and TMA stores
  const uint8_t* scale;   // [E, Wn, Wk / 16] e4m3 bytes
  const float* pts;       // [E]
  const int4* passes;     // (first row block, expert, rows, row blocks) of every pass
  const int* n_pass;
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

// One pass: up to 256 consecutive rows of one expert against one 256-column tile of its weights. Every role walks this CTA pair's
// tiles and requests the next tile's pass while it works on the current one: the trip to L2 at the start of a pass, in each of the
// roles that wait for one another, is a gap of the whole pipeline otherwise.
struct Tiles {
  const W4Params& p;
  const int num_n, step, total;
  int tile;
  int4 ps, ahead;
  AXB_DEVICE Tiles(const W4Params& p_, int num_n_, int total_, int first, int step_)
      : p(p_), num_n(num_n_), step(step_), total(total_), tile(first), ps(get(first)), ahead(get(first + step_)) {}
  AXB_DEVICE int4 get(int t) const {
    int4 r = make_int4(0, 0, 0, 0);
    if (t < total) r = __ldg(p.passes + t / num_n);
    if (!AXB_INDEX_OK(AXB_SITE_W4A16_EXPERT, r.y, p.E)) r.y = 0;        // checked build: recorded, then a valid expert
    return r;
  }
  AXB_DEVICE bool live() const { return tile < total; }
  AXB_DEVICE int col0() const { return (tile % num_n) * BN; }
  AXB_DEVICE void next() {
    tile += step;
    ps = ahead;
    ahead = get(tile + step);
  }
};
// Rows of a pass that enter the product: whole 32-row groups, half of them staged by each CTA.
AXB_DEVICE int pass_cols(const int4& ps) { return (ps.z + 31) & ~31; }

template <bool DX>
__global__ void __launch_bounds__(W4_THREADS, 1)
    grouped_w4a16_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmXs,
                         const __grid_constant__ CUtensorMap tmX2, const __grid_constant__ CUtensorMap tmX2s,
                         const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmW2,
                         const __grid_constant__ CUtensorMap tmC, const W4Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sX = smem;                                   // [slot][<= 128 rows x 64]
  uint8_t* sW = sX + SX * X_BYTES;                      // [slot][128 weight columns x 64]
  uint8_t* sRaw = sW + SW * W_BYTES;
  uint8_t* sEpi = sRaw + SR * RAW_BYTES;                // per epilogue warp: two slots of 32 rows x 32 columns
  uint8_t* sTab = sEpi + 4 * EPI_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sTab + CGROUPS * TAB_BYTES);
  // x_full, w_full and tempty are used in rank 0 only and hear from both CTAs
  uint64_t* x_full = bars;                      // rows landed
  uint64_t* x_empty = x_full + SX;              // their MMAs retired
  uint64_t* w_full = x_empty + SX;              // decoded tiles in place (one arrival per warp of the groups; LoRA tiles by TMA)
  uint64_t* w_empty = w_full + SW;
  uint64_t* r_full = w_empty + SW;              // packed weights landed
  uint64_t* r_empty = r_full + SR;              // read by their group
  uint64_t* tfull_bar = r_empty + SR;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  const int num_n = (p.N + BN - 1) / BN;
  const int nk_main = (p.K + BK - 1) / BK, nk_ext = (p.K2 + BK - 1) / BK;
  const int nk = nk_main + nk_ext;
  const int total = *p.n_pass * num_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < SX; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1);
    }
    for (int s = 0; s < SW; ++s) {
      mbar_init(&w_full[s], 2 * CG_WARPS);
      mbar_init(&w_empty[s], 1);
    }
    for (int s = 0; s < SR; ++s) {
      mbar_init(&r_full[s], 1);
      mbar_init(&r_empty[s], CG_WARPS);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull_bar[s], 1);
      mbar_init(&tempty_bar[s], 8);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmQ);
  }
  if (warp == 2) {
    tmem_alloc_pair(tmem_slot, 512);   // two accumulators of 256 columns
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // barriers of both CTAs are initialised before any remote arrival or TMA credit
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ rows
    Ring<SX> rx;
    bool ok = true;
    for (Tiles t(p, num_n, total, cluster_id, n_clusters); t.live() && ok; t.next()) {
      const int half = pass_cols(t.ps) / 2, row0 = t.ps.x * 128 + rank * half;
      for (int kb = 0; kb < nk; ++kb, rx.next()) {
        if (!warp_all(wait_sleeping(&x_empty[rx.slot], rx.phase ^ 1, 40, p.status, AXB_TIMEOUT_EMPTY))) {
          ok = false;
          break;
        }
        const bool ext = kb >= nk_main;
        const int k0 = (ext ? kb - nk_main : kb) * BK;
        uint8_t* dst = sX + rx.slot * X_BYTES;
        const uint32_t fb = mapa_u32(smem_u32(&x_full[rx.slot]), 0);    // the partner's loads credit the leader's barrier
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&x_full[rx.slot], 2 * half * 128);
          if (half == 128) {
            tma_load_2d_pair(dst, ext ? &tmX2 : &tmX, fb, k0, row0);
          } else {
            const CUtensorMap* m = ext ? &tmX2s : &tmXs;
            for (int r = 0; r < half; r += 16) tma_load_2d_pair(dst + r * 128, m, fb, k0, row0 + r);
          }
        }
        __syncwarp();
      }
    }
  } else if (warp == W4_THREADS / 32 - 1) {
    // ------------------------------------------------------------ packed weights
    Ring<SR> rr;
    bool ok = true;
    for (Tiles t(p, num_n, total, cluster_id, n_clusters); t.live() && ok; t.next()) {
      const int n0 = t.col0() + rank * 128;
      for (int kb = 0; kb < nk; ++kb, rr.next()) {
        if (!warp_all(mbar_wait(&r_empty[rr.slot], rr.phase ^ 1, p.status, AXB_TIMEOUT_EMPTY))) {
          ok = false;
          break;
        }
        if (kb >= nk_main) {          // a LoRA block has no packed weights: its slot only keeps the order
          if (elect_one()) mbar_arrive(&r_full[rr.slot]);
        } else if (elect_one()) {
          mbar_expect_tx(&r_full[rr.slot], RAW_BYTES);
          if (!DX) tma_load_3d(sRaw + rr.slot * RAW_BYTES, &tmQ, &r_full[rr.slot], kb * (BK / 2), n0, t.ps.y);   // [128 n, 32 B of k]
          else tma_load_3d(sRaw + rr.slot * RAW_BYTES, &tmQ, &r_full[rr.slot], n0 / 2, kb * BK, t.ps.y);         // [64 k, 64 B of n]
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issue (rank 0, for both CTAs)
    if (rank == 0) {
      const uint64_t da_base = DX ? make_smem_desc_sw128(smem_u32(sW), 8192, 1024) : make_smem_desc_sw128(smem_u32(sW), 16, 1024);
      const uint64_t db_base = make_smem_desc_sw128(smem_u32(sX), 16, 1024);
      Ring<SX> rx;
      Ring<SW> rw;
      int it = 0;
      bool ok = true;
      for (Tiles t(p, num_n, total, cluster_id, n_clusters); t.live() && ok; t.next(), ++it) {
        const uint32_t idesc = make_idesc_bf16(256, pass_cols(t.ps), DX ? 1 : 0, 0);
        const int acc = it & 1;
        if (!warp_all(mbar_wait_partner(&tempty_bar[acc], ((it >> 1) & 1) ^ 1, p.status, AXB_TIMEOUT_TMEM_EMPTY))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int kb = 0; kb < nk; ++kb, rx.next(), rw.next()) {
          if (!warp_all(mbar_wait_spin(&x_full[rx.slot], rx.phase, p.status, AXB_TIMEOUT_FULL) &&
                        mbar_wait_partner(&w_full[rw.slot], rw.phase, p.status, AXB_TIMEOUT_FULL))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t da = da_base + (uint32_t)(rw.slot * (W_BYTES / 16)), db = db_base + (uint32_t)(rx.slot * (X_BYTES / 16));
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              umma_f16_pair(d_tmem, da + kk * (DX ? 2048 / 16 : 32 / 16), db + kk * 2, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
            umma_commit_pair_mc(&x_empty[rx.slot]);
            umma_commit_pair_mc(&w_empty[rw.slot]);
            if (kb == nk - 1) umma_commit_pair_mc(&tfull_bar[acc]);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp >= 6) {
    // ------------------------------------------------------------ converters: packed tile -> bf16 tile
    // A k block of this CTA is 256 units of 16 packed bytes (32 codes, 2 scale groups); thread t of a group takes units t, t + 128
    // Unit ct lies at raw + ct * 16 and becomes four 16-byte chunks of the swizzled bf16 tile.
    //   FWD: raw tile [128 n][32 B]: weight row n0 + ct / 2, codes 32 * (ct & 1) .. + 31 of k block kb
    //        -> K-major row ct / 2, chunks 4 * (ct & 1) .. + 3.
    //   DX : raw tile [64 wn][64 B]: weight row kb * 64 + ct / 4, columns n0 + 64 * half + 32 * part .. + 31
    //        (half = (ct >> 1) & 1, part = ct & 1) -> MN-major chunk block `half`, row ct / 4, chunks 4 * part .. + 3.
    // Shared-memory accesses to the tiles are conflict free: the loads are contiguous, and the eight lanes of a store phase
    // hit eight different 16-byte chunk positions (rows differ in swizzle bits 0-1 or bit 0, `part` flips bit 2,
    // and in dX the odd half walks its chunks in the order 2, 3, 0, 1, which flips bit 1).
    const int cw = warp - 6, grp = cw / CG_WARPS, gt = (cw % CG_WARPS) * 32 + lane;
    const long long sc_row_bytes = p.Wk / 16;
    const int part = gt & 1, half = DX ? ((gt >> 1) & 1) : 0;      // the same for all units of a thread
    const uint32_t wf0 = mapa_u32(smem_u32(w_full), 0);
    auto arrive_full = [&](int slot) {
      if (rank == 0) mbar_arrive(&w_full[slot]);
      else mbar_arrive_partner(wf0 + slot * 8);
    };
    // This group's k blocks are every fourth of the whole sequence; `it` is the one at hand, `nx` the next, `t` walks with `nx`.
    struct At {
      int kb, e, n0;
      bool live;
    };
    Tiles t(p, num_n, total, cluster_id, n_clusters);
    auto settle = [&](int kb) {        // the k block `kb` of the pass that `t` stands at, or of one behind it
      while (kb >= nk && t.live()) kb -= nk, t.next();
      return At{kb, t.ps.y, t.col0() + rank * 128, t.live()};
    };
    // the two E4M3 bytes of each unit, requested one turn (four k blocks) ahead and looked at when they are needed
    auto load_scales = [&](const At& a, uint32_t (&out)[CG_UNITS]) {
      const uint8_t* base = p.scale + (long long)a.e * p.Wn * sc_row_bytes;
#pragma unroll
      for (int u = 0; u < CG_UNITS; ++u) {
        out[u] = 0u;
        const int ct = gt + u * (256 / CG_UNITS);
        if (!a.live || a.kb >= nk_main) continue;
        if (!DX) {
          const int n = a.n0 + (ct >> 1);
          if (n < p.Wn) out[u] = __ldg(reinterpret_cast<const unsigned short*>(base + (long long)n * sc_row_bytes + a.kb * 4 + part * 2));
        } else {
          const int k0 = a.n0 + half * 64 + part * 32, wn = a.kb * BK + (ct >> 2);
          if (k0 < p.Wk && wn < p.Wn) out[u] = __ldg(reinterpret_cast<const unsigned short*>(base + (long long)wn * sc_row_bytes + k0 / 16));
        }
      }
    };
    uint4* table = reinterpret_cast<uint4*>(sTab + grp * TAB_BYTES);
    auto products = [&](uint32_t byte, float g) -> uint4 {     // a negative scale is legal, if nobody writes one
      return byte < 128 ? table[byte] : make_lut(e4m3_to_float(byte) * g);
    };
    At it = settle(grp);
    uint32_t cur[CG_UNITS], nxt[CG_UNITS];
    load_scales(it, cur);
    float g = it.live ? p.pts[it.e] : 0.f;
    int table_e = -1;
    bool dead = false;    // a wait ran out: the warp walks on without work, because its group still meets it at the table's barriers
    for (uint32_t at = grp; it.live; at += CGROUPS) {
      const At nx = settle(it.kb + CGROUPS);
      load_scales(nx, nxt);
      const float g_next = nx.live ? p.pts[nx.e] : 0.f;
      if (it.e != table_e) {
        // A third of the decode's integer work went into these products when each scale group made its own: one table of an expert's
        // 128 scale magnitudes serves every k block of the pass.
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * CG_WARPS) : "memory");
        for (int b = gt; b < 128; b += 32 * CG_WARPS) table[b] = make_lut(e4m3_to_float((uint32_t)b) * g);
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * CG_WARPS) : "memory");
        table_e = it.e;
      }
      const int rslot = (int)(at % SR), wslot = (int)(at % SW);
      uint8_t* w_tile = sW + wslot * W_BYTES;
      const uint32_t wphase = (at / SW) & 1, rphase = (at / SR) & 1;
      if (!dead) dead = !warp_all(mbar_wait(&r_full[rslot], rphase, p.status, AXB_TIMEOUT_FULL));
      uint4 w[CG_UNITS];
      if (!dead && it.kb < nk_main) {
#pragma unroll
        for (int u = 0; u < CG_UNITS; ++u)
          w[u] = *reinterpret_cast<const uint4*>(sRaw + rslot * RAW_BYTES + (gt + u * (256 / CG_UNITS)) * 16);
      }
      if (!dead) dead = !warp_all(mbar_wait_spin(&w_empty[wslot], wphase ^ 1, p.status, AXB_TIMEOUT_EMPTY));
      if (!dead && it.kb < nk_main) {
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
          uint8_t* dst_row = w_tile + half * 8192 + r * 128;
          const uint4 t0 = products(sc2 & 0xFF, g), t1 = products(sc2 >> 8, g);
          *reinterpret_cast<uint4*>(dst_row + ((pos ^ 0) << 4)) = decode8(w[u].x, t0);
          *reinterpret_cast<uint4*>(dst_row + ((pos ^ 1) << 4)) = decode8(w[u].y, t0);
          *reinterpret_cast<uint4*>(dst_row + ((pos ^ 2) << 4)) = decode8(w[u].z, t1);
          *reinterpret_cast<uint4*>(dst_row + ((pos ^ 3) << 4)) = decode8(w[u].w, t1);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          arrive_full(wslot);
          mbar_arrive(&r_empty[rslot]);
        }
      } else if (!dead) {                         // the LoRA tile comes by TMA, on the group's first arrival
        if (lane == 0) {
          mbar_arrive(&r_empty[rslot]);
          if (cw % CG_WARPS == 0) {
            const int ka = (it.kb - nk_main) * BK;
            const uint32_t wf = wf0 + wslot * 8;
            if (rank == 0) mbar_expect_tx(&w_full[wslot], 2 * W_BYTES);
            else mbar_arrive_partner(wf);
            if (!DX) {
              tma_load_3d_pair(w_tile, &tmW2, wf, ka, it.n0, it.e);
            } else {
              tma_load_3d_pair(w_tile, &tmW2, wf, it.n0, ka, it.e);
              tma_load_3d_pair(w_tile + 8192, &tmW2, wf, it.n0 + 64, ka, it.e);
            }
          } else {
            arrive_full(wslot);
          }
        }
        __syncwarp();
      }
#pragma unroll
      for (int u = 0; u < CG_UNITS; ++u) cur[u] = nxt[u];
      it = nx;
      g = g_next;
    }
  } else {
    // ------------------------------------------------------------ epilogue warps 2..5
    // The accumulator is transposed: lane = weight column, TMEM column = row of the pass. Neighbouring lanes trade one of two rows,
    // so that a row's 32 columns leave as 64 contiguous bytes of a staging tile.
    const int lg = warp & 3;
    uint8_t* stage = sEpi + lg * EPI_BYTES;
    const uint32_t pair_sel = (lane & 1) ? 0x3276u : 0x5410u;
    int it = 0, slot = 0;
    bool ok = true;
    for (Tiles t(p, num_n, total, cluster_id, n_clusters); t.live() && ok; t.next(), ++it) {
      const int4 ps = t.ps;
      const int col0 = t.col0() + rank * 128 + lg * 32;      // this warp's columns
      const int cols = pass_cols(ps);
      const int acc = it & 1;
      ok = warp_all(wait_sleeping(&tfull_bar[acc], (it >> 1) & 1, 200, p.status, AXB_TIMEOUT_TMEM_FULL));
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_addr = tmem_base + (uint32_t(lg * 32) << 16) + acc * 256;
      // the rows that pad a block are written too, as zeros: one staging tile of them serves all their stores
      bool zeros = false;
#pragma unroll 1
      for (int c = 0; c < ps.w * 4; ++c) {
        uint32_t r[32];
        if (c * 32 < cols) {
          tmem_ld_32x32(t_addr + c * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (col0 >= p.N) continue;
        const long long row = (long long)ps.x * 128 + c * 32;
        if (p.tma_store) {
          if (!zeros) {
            slot ^= 1;
            if (lane == 0) bulk_wait_group_read<1>();   // the store that last read this slot is done with it
            __syncwarp();
            uint32_t* mine = reinterpret_cast<uint32_t*>(stage + slot * (EPI_BYTES / 2) + (lane & 1) * 64 + (lane >> 1) * 4);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const uint32_t u = pack_bf16x2(__uint_as_float(r[2 * i]) * p.alpha, __uint_as_float(r[2 * i + 1]) * p.alpha);
              mine[i * 32] = prmt(u, __shfl_xor_sync(0xffffffffu, u, 1), pair_sel);
            }
            fence_proxy_async_smem();
            __syncwarp();
            zeros = c * 32 >= cols;
          }
          if (lane == 0) {
            tma_store_2d(&tmC, stage + slot * (EPI_BYTES / 2), col0, (int)row);
            bulk_commit_group();
          }
        } else if (col0 + lane < p.N) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float v = __uint_as_float(r[i]) * p.alpha;
            const long long at = (row + i) * p.ldc + col0 + lane;
            if (p.out_mode == 0) reinterpret_cast<__nv_bfloat16*>(p.C)[at] = __float2bfloat16(v);
            else reinterpret_cast<float*>(p.C)[at] = v;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tempty_bar[acc]), 0));
    }
    if (lane == 0) bulk_wait_group<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();   // neither CTA leaves while its partner still signals it or reads its tiles
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <bool DX>
int launch_w4a16(const CUtensorMap& tX, const CUtensorMap& tXs, const CUtensorMap& tX2, const CUtensorMap& tX2s, const CUtensorMap& tQ,
                 const CUtensorMap& tW2, const CUtensorMap& tC, const W4Params& p, int grid, cudaStream_t st) {
  static std::atomic<unsigned long long> allowed{0};
  if (const int rc = axb_allow_smem((const void*)grouped_w4a16_kernel<DX>, W4_SMEM, allowed)) return rc;
  AxbLaunch l(dim3(grid), W4_THREADS, W4_SMEM, st, 2, false);
  return (int)cudaLaunchKernelEx(&l.cfg, grouped_w4a16_kernel<DX>, tX, tXs, tX2, tX2s, tQ, tW2, tC, p);
}

}  // namespace

// A [max_blocks * 128, Ka] bf16 (lda); qdata [E, Wn, Wk/2] uint8, scale [E, Wn, Wk/16] e4m3 bytes, pts [E] fp32.
//   trans_w = 0 (forward):        Ka = Wk, C [rows, Wn];  A2 [rows, K2], W2 [E, Wn, K2] (bf16, optional)
//   trans_w = 1 (input gradient): Ka = Wn, C [rows, Wk];  A2 [rows, K2], W2 [E, K2, Wk] (bf16, optional)
// Wk must be a multiple of 64, Wn a multiple of 8; out_mode 0 bf16 / 1 fp32. passes int32 [<= max_blocks, 4] (16-byte aligned): first
// row block, expert, rows in use, row blocks (1 or 2); rows of a block beyond those in use come out as zeros. n_pass: their number.
extern "C" int axb_grouped_gemm_w4a16(const void* A, long long lda, const void* qdata, const void* scale, const float* pts,
                                      const void* A2, long long lda2, const void* W2, void* C, long long ldc, int E,
                                      int Wn, int Wk, int K2, int trans_w, float alpha, int out_mode,
                                      const int* passes, const int* n_pass, int max_blocks, int* status,
                                      void* stream) {
  if (max_blocks <= 0 || Wn <= 0 || Wk <= 0) return 0;
  if ((lda & 7) || (Wk & 63) || (Wn & 7) || (K2 > 0 && ((lda2 & 7) || (K2 & 7))) || out_mode < 0 || out_mode > 1) return -2;
  if (reinterpret_cast<uintptr_t>(passes) & 15) return -2;
  const unsigned long long rows = (unsigned long long)max_blocks * 128;
  const int Ka = trans_w ? Wn : Wk, N = trans_w ? Wk : Wn;
  CUtensorMap tX, tXs, tX2, tX2s, tQ, tW2, tC;
  int rc = axb_make_tmap_2d(&tX, A, rows, Ka, lda, 128, 64) | axb_make_tmap_2d(&tXs, A, rows, Ka, lda, 16, 64);
  rc |= trans_w ? make_tmap_u8_3d(&tQ, qdata, E, Wn, Wk / 2, 64, 64) : make_tmap_u8_3d(&tQ, qdata, E, Wn, Wk / 2, 128, 32);
  if (K2 > 0) {
    rc |= axb_make_tmap_2d(&tX2, A2, rows, K2, lda2, 128, 64) | axb_make_tmap_2d(&tX2s, A2, rows, K2, lda2, 16, 64);
    rc |= trans_w ? axb_make_tmap_3d(&tW2, W2, E, K2, Wk, Wk, (unsigned long long)Wk * K2, 64, 64)
                  : axb_make_tmap_3d(&tW2, W2, E, Wn, K2, K2, (unsigned long long)Wn * K2, 128, 64);
  } else {
    tX2 = tX2s = tW2 = tX;
  }
  const bool tma_store = out_mode == 0 && (ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  tC = tX;
  if (tma_store) rc |= axb_make_tmap_2d(&tC, C, rows, N, ldc, 32, 32, 2, false);
  if (rc) return -4;
  W4Params p = {};
  p.tma_store = tma_store;
  p.N = N; p.K = Ka; p.K2 = K2 > 0 ? K2 : 0; p.Wn = Wn; p.Wk = Wk; p.E = E;
  p.C = C; p.ldc = ldc; p.alpha = alpha; p.out_mode = out_mode;
  p.scale = reinterpret_cast<const uint8_t*>(scale); p.pts = pts;
  p.passes = reinterpret_cast<const int4*>(passes); p.n_pass = n_pass; p.status = status;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long max_tiles = (long long)max_blocks * ((N + BN - 1) / BN);
  const int grid = 2 * max_tiles < sms ? (int)(2 * max_tiles) : sms & ~1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return trans_w ? launch_w4a16<true>(tX, tXs, tX2, tX2s, tQ, tW2, tC, p, grid, st)
                 : launch_w4a16<false>(tX, tXs, tX2, tX2s, tQ, tW2, tC, p, grid, st);
}
