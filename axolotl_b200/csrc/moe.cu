// Mixture-of-experts support kernels for sm_100a.
//
//  * nvfp4_dequant     : packed E2M1 nibbles x E4M3 block scales (16 elements) x fp32 per-tensor
//                        scale -> bf16 rows, for the frozen NVFP4 expert weights (storage contract
//                        of src/axolotl/integrations/kernels/libs/scattermoe_lora/dequant_grouped.py:63-111).
//  * ep_gather_rows    : expert-parallel DISPATCH. Every destination rank pulls the token rows
//                        routed to its experts straight out of the source ranks' symmetric
//                        activation buffers with peer loads over NVLink (row list: source rank +
//                        source row), writing them expert-sorted into a local buffer.
//  * ep_scatter_add    : expert-parallel COMBINE. Expert outputs are multiplied by their routing
//                        weight and reduce-added (bf16x2 atomics over NVLink) into the source
//                        rank's output buffer at the token's row.
//  * peer_put_i32      : routing metadata exchange (plain peer stores).
// Together they replace DeepEP's dispatch / combine + host barrier of the reference
// (src/axolotl/integrations/expert_parallel/experts_fn.py:185-342).
#include "axb_common.cuh"

namespace {

// bf16 bit patterns of the 8 E2M1 magnitudes {0, .5, 1, 1.5, 2, 3, 4, 6}, 16 bits each, held in two
// 64-bit registers: a lookup is a shift (no memory access, no divergence).
constexpr unsigned long long kE2M1Lo = 0x3fc03f803f000000ull;  // 1.5, 1.0, 0.5, 0.0
constexpr unsigned long long kE2M1Hi = 0x40c0408040404000ull;  // 6.0, 4.0, 3.0, 2.0

AXB_DEVICE float e2m1_to_float(uint32_t code) {
  const unsigned long long tbl = (code & 4) ? kE2M1Hi : kE2M1Lo;
  const uint32_t bits = (uint32_t)(tbl >> ((code & 3) * 16)) & 0xFFFFu;
  return __uint_as_float((bits | ((code & 8) << 12)) << 16);
}

AXB_DEVICE float e4m3_to_float(uint8_t v) {
  const uint32_t sign = (v >> 7) & 1, exp = (v >> 3) & 0xF, man = v & 7;
  float f;
  if (exp == 0) f = ldexpf((float)man, -9);                 // subnormal: man * 2^-3 * 2^-6
  else if (exp == 15 && man == 7) f = __int_as_float(0x7fc00000);
  else f = __uint_as_float(((exp + 120u) << 23) | (man << 20));
  return sign ? -f : f;
}

// One thread per 16 bytes of packed codes (32 values = two 16-element scale blocks): 16-byte
// loads, four 16-byte stores; a warp reads 512 contiguous bytes and writes 2 KB contiguous.
__global__ void nvfp4_dequant_kernel(const uint8_t* __restrict__ q, const uint8_t* __restrict__ scale,
                                     const float* __restrict__ pts, __nv_bfloat16* __restrict__ out,
                                     long long n_blocks, long long blocks_per_pts,
                                     const int* __restrict__ active) {
  const long long n_pairs = n_blocks >> 1;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n_pairs;
       t += (long long)gridDim.x * blockDim.x) {
    const long long b = t * 2;
    const long long mat = b / blocks_per_pts;
    if (active && active[mat] == 0) continue;   // selective dequant: no row is routed to this expert
    const float g = pts[mat];
    const unsigned short sc = *reinterpret_cast<const unsigned short*>(scale + b);
    const float s0 = e4m3_to_float(sc & 0xFF) * g, s1 = e4m3_to_float(sc >> 8) * g;
    const uint4 packed = *reinterpret_cast<const uint4*>(q + b * 8);
    const uint32_t w[4] = {packed.x, packed.y, packed.z, packed.w};
    uint32_t o[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float s = i < 2 ? s0 : s1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t byte = (w[i] >> (8 * j)) & 0xFF;
        o[i * 4 + j] = pack_bf16x2(e2m1_to_float(byte & 0xF) * s, e2m1_to_float(byte >> 4) * s);
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + b * 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
  }
  // odd trailing block (K/16 odd for a single row) is handled by the last thread
  if ((n_blocks & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    const long long b = n_blocks - 1;
    const float s = e4m3_to_float(scale[b]) * pts[b / blocks_per_pts];
    for (int i = 0; i < 8; ++i) {
      const uint32_t byte = q[b * 8 + i];
      out[b * 16 + 2 * i] = __float2bfloat16(e2m1_to_float(byte & 0xF) * s);
      out[b * 16 + 2 * i + 1] = __float2bfloat16(e2m1_to_float(byte >> 4) * s);
    }
  }
}

// ---- Layout of a routed batch: the T * k slots sorted by expert, every expert's rows padded to whole 128-row blocks, slots of
// an expert in slot order. Three launches (count, place, scatter) instead of two dozen tensor operations around a sort, whose
// issue cost exceeded the expert GEMMs of a short batch.
constexpr int RL_T = 1024;        // slots per block of the counting and scattering kernels
constexpr int RL_MAX_E = 1024;

__global__ void __launch_bounds__(RL_T) route_count_kernel(const long long* __restrict__ expert, int* __restrict__ hist, int n, int E) {
  extern __shared__ int h[];      // [E]
  for (int e = threadIdx.x; e < E; e += RL_T) h[e] = 0;
  __syncthreads();
  const int i = blockIdx.x * RL_T + threadIdx.x;
  if (i < n) {
    const long long e = expert[i];
    if (e >= 0 && e < E) atomicAdd(&h[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += RL_T) hist[(long long)blockIdx.x * E + e] = h[e];
}

// Sum of `own` over the threads before this one; warp_sum: 32 words of shared memory. Every thread of a block of 1024 calls it.
AXB_DEVICE unsigned long long sum_before(unsigned long long own, unsigned long long* warp_sum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    unsigned long long v = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    warp_sum[lane] = v;
  }
  __syncthreads();
  return incl - own + (warp ? warp_sum[warp - 1] : 0);
}

// hist[b][e] becomes the padded row of the first slot of expert e in block b
__global__ void __launch_bounds__(RL_MAX_E) route_place_kernel(int* __restrict__ hist, int blocks, int E, int max_blocks,
                                                               int* __restrict__ seg_start, int* __restrict__ seg_rows,
                                                               int* __restrict__ blk_expert, int* __restrict__ n_blocks,
                                                               int4* __restrict__ passes, int* __restrict__ n_pass) {
  __shared__ unsigned long long warp_sum[32];
  __shared__ int first[RL_MAX_E + 1];     // first 128-row block of every expert
  const int e = threadIdx.x;
  int count = 0;
  if (e < E) {
#pragma unroll 8
    for (int b = 0; b < blocks; ++b) count += hist[(long long)b * E + e];
  }
  // running sums over the experts: blocks of 128 rows (low word), passes of the NVFP4 GEMM over two blocks (high word)
  const int nb = (count + 127) / 128, np = (nb + 1) / 2;
  const unsigned long long before = sum_before((unsigned long long)np << 32 | (unsigned)nb, warp_sum);
  const int start = (int)(unsigned)before, pass0 = (int)(before >> 32);
  if (e < E) {
    first[e] = start;
    if (e == E - 1) {
      first[E] = start + nb;
      *n_blocks = start + nb;
      *n_pass = pass0 + np;
    }
    for (int j = 0; j < np; ++j) passes[pass0 + j] = make_int4(start + 2 * j, e, min(256, count - 256 * j), min(2, nb - 2 * j));
    seg_start[e] = start * 128;
    seg_rows[e] = nb * 128;
    int row = start * 128;
    for (int b = 0; b < blocks; ++b) {
      const int c = hist[(long long)b * E + e];
      hist[(long long)b * E + e] = row;
      row += c;
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < max_blocks; b += RL_MAX_E) {   // the expert whose blocks hold b; the last one beyond them
    int lo = 0, hi = E - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (first[mid + 1] > b) hi = mid;
      else lo = mid + 1;
    }
    blk_expert[b] = lo;
  }
}

// The passes of the NVFP4 grouped GEMM for a layout given by its rows per expert (any number of experts). A layout that was sized for
// fewer blocks than its rows need ends at max_blocks; a pass's first block grows with the pass, so those that begin before it are a
// prefix of the table. Bound: its launch, 10 to 13 us with the two allocations; as tensor operations with a sort the table took 180 to
// 195 us of the host, half of a forward product over 2664 rows of 128 experts (layout and product 454 -> 300 us, 65536 rows 591 -> 486).
__global__ void __launch_bounds__(RL_MAX_E) group_passes_kernel(const long long* __restrict__ counts, int E, int max_blocks,
                                                                int4* __restrict__ passes, int* __restrict__ n_pass) {
  __shared__ unsigned long long warp_sum[32];
  __shared__ unsigned long long done;       // blocks (low word) and passes (high word) of the experts before this chunk
  __shared__ int n;
  if (threadIdx.x == 0) done = 0, n = 0;
  __syncthreads();
  for (int e0 = 0; e0 < E; e0 += RL_MAX_E) {
    const int e = e0 + threadIdx.x;
    const int count = e < E ? (int)counts[e] : 0, nb = (count + 127) / 128, np = (nb + 1) / 2;
    const unsigned long long own = (unsigned long long)np << 32 | (unsigned)nb;
    const unsigned long long before = done + sum_before(own, warp_sum);
    const int start = (int)(unsigned)before, pass0 = (int)(before >> 32);
    int mine = 0;
    for (; mine < np && start + 2 * mine < max_blocks; ++mine) {
      const int b = start + 2 * mine, blocks = min(min(2, nb - 2 * mine), max_blocks - b);
      passes[pass0 + mine] = make_int4(b, e, min(blocks * 128, count - 256 * mine), blocks);
    }
    if (mine) atomicAdd(&n, mine);
    __syncthreads();                        // everyone has read `done`
    if (threadIdx.x == RL_MAX_E - 1) done = before + own;
    __syncthreads();
  }
  if (threadIdx.x == 0) *n_pass = n;
}

__global__ void __launch_bounds__(RL_T) route_scatter_kernel(const long long* __restrict__ expert, const int* __restrict__ base,
                                                             int* __restrict__ slot_row, int* __restrict__ row_slot, int n, int E,
                                                             int* status) {
  extern __shared__ unsigned short c[];   // [32 warps][E]: slots of the expert in the warps before
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 32 * E; i += RL_T) c[i] = 0;
  __syncthreads();
  const int i = blockIdx.x * RL_T + threadIdx.x;
  const long long e64 = i < n ? expert[i] : -1;
  const int e = i < n && axb_index_checked(AXB_SITE_ROUTE_EXPERT, e64, E, true, status) ? (int)e64 : -1;
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int rank = __popc(same & ((1u << lane) - 1u));
  if (e >= 0 && rank == 0) c[warp * E + e] = (unsigned short)__popc(same);
  __syncthreads();
  for (int q = threadIdx.x; q < E; q += RL_T) {
    unsigned run = 0;
#pragma unroll 8
    for (int w = 0; w < 32; ++w) {
      const unsigned v = c[w * E + q];
      c[w * E + q] = (unsigned short)run;
      run += v;
    }
  }
  __syncthreads();
  if (e >= 0) {
    const int row = base[(long long)blockIdx.x * E + e] + c[warp * E + e] + rank;
    slot_row[i] = row;
    row_slot[row] = i;
  } else if (i < n) {
    slot_row[i] = -1;             // no such expert: combined as zero
  }
}

// Local dispatch: out[r, :] = scale * x[token of row r, :], zeros in pad rows. Row r holds slot row_slot[r] (-1: a pad row), the
// slots of token t are t * k .. t * k + k - 1, the scale is slot_scale[slot] (null: 1). One warp per row; eight vectors of a row
// are requested before the first is stored.
__global__ void moe_dispatch_rows_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ row_slot,
                                         const float* __restrict__ slot_scale, __nv_bfloat16* __restrict__ out,
                                         long long n_rows, int width, int k) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = w; r < n_rows; r += n_warps) {
    const int id = row_slot[r];
    __nv_bfloat16* d = out + r * width;
    if (id < 0) {
      for (int c = lane * 8; c < width; c += 256) *reinterpret_cast<uint4*>(d + c) = make_uint4(0, 0, 0, 0);
      continue;
    }
    const __nv_bfloat16* s = x + (long long)(id / k) * width;
    const float g = slot_scale ? slot_scale[id] : 1.f;
    for (int c0 = 0; c0 < width; c0 += 8 * 256) {
      uint4 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int c = c0 + q * 256 + lane * 8;
        v[q] = c < width ? *reinterpret_cast<const uint4*>(s + c) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int c = c0 + q * 256 + lane * 8;
        if (c >= width) break;
        if (slot_scale) {
          uint32_t in[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_bf16x2(in[e]);
            in[e] = pack_bf16x2(f.x * g, f.y * g);
          }
          v[q] = make_uint4(in[0], in[1], in[2], in[3]);
        }
        *reinterpret_cast<uint4*>(d + c) = v[q];
      }
    }
  }
}

// Local combine: out[t, :] = sum_j w[t, j] * ys[slot_row[t, j], :] (fp32 accumulation in slot order, no atomics; a slot
// without a row, -1, is zero). One warp per (token, 256 columns); the rows of eight slots are requested together (a warp per token with one load at a time took 30 us
// for 333 tokens).
__global__ void moe_combine_rows_kernel(const __nv_bfloat16* __restrict__ ys, const int* __restrict__ slot_row,
                                        const float* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                        long long n_tokens, int k, int width) {
  const int lane = threadIdx.x & 31;
  const int chunks = (width + 255) / 256;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long it = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < n_tokens * chunks; it += n_warps) {
    const long long t = it / chunks;
    const int c = (int)(it - t * chunks) * 256 + lane * 8;
    const bool in_row = c < width;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j0 = 0; j0 < k; j0 += 8) {
      const int mine = j0 + (lane & 7);
      const int my_row = mine < k ? slot_row[t * k + mine] : -1;
      const float my_w = my_row >= 0 ? (w ? w[t * k + mine] : 1.f) : 0.f;
      uint4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = __shfl_sync(0xffffffffu, my_row, j);
        v[j] = in_row && r >= 0 ? *reinterpret_cast<const uint4*>(ys + (long long)r * width + c) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float g = __shfl_sync(0xffffffffu, my_w, j);
        if (j0 + j >= k) break;
        const uint32_t in[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = unpack_bf16x2(in[e]);
          acc[2 * e] += g * f.x;
          acc[2 * e + 1] += g * f.y;
        }
      }
    }
    if (in_row)
      *reinterpret_cast<uint4*>(out + t * width + c) =
          make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                     pack_bf16x2(acc[6], acc[7]));
  }
}

// dw[t, j] = <dy[t, :], ys[slot_row[t, j], :]>  (gradient of the routing weights; one warp per slot, eight vectors of each row
// in flight)
__global__ void moe_combine_dw_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ ys,
                                      const int* __restrict__ slot_row, float* __restrict__ dw, long long n_slots,
                                      int k, int width) {
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long sl = wid; sl < n_slots; sl += n_warps) {
    const __nv_bfloat16* a = dy + (sl / k) * width;
    const int row = slot_row[sl];                 // -1: no row, the gradient is zero
    const __nv_bfloat16* b = ys + (long long)row * width;
    float acc = 0.f;
    for (int c0 = lane * 8; c0 < width; c0 += 8 * 256) {
      uint4 va[8], vb[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int c = c0 + q * 256;
        va[q] = vb[q] = make_uint4(0, 0, 0, 0);
        if (c < width && row >= 0) {
          va[q] = *reinterpret_cast<const uint4*>(a + c);
          vb[q] = *reinterpret_cast<const uint4*>(b + c);
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t ia[4] = {va[q].x, va[q].y, va[q].z, va[q].w}, ib[4] = {vb[q].x, vb[q].y, vb[q].z, vb[q].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 fa = unpack_bf16x2(ia[e]), fb = unpack_bf16x2(ib[e]);
          acc += fa.x * fb.x + fa.y * fb.y;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) dw[sl] = acc;
  }
}

struct PeerPtrs8 {
  unsigned long long p[8];
};

// out[i, :] = scale(i) * src_rank(i).buffer[src_row(i), :]   (one warp per row, 16-byte vectors).
// src_rank(i) < 0 marks a pad row of the expert-sorted layout: it is written as zeros.
// Optionally dot_out[i] = <unscaled gathered row, dot_with[i, :]> (gradient of the routing weight).
__global__ void ep_gather_rows_kernel(PeerPtrs8 src, const int* __restrict__ src_rank,
                                      const int* __restrict__ src_row, const float* __restrict__ scale,
                                      const __nv_bfloat16* __restrict__ dot_with, float* __restrict__ dot_out,
                                      __nv_bfloat16* __restrict__ out, long long n_rows, int width, long long src_ld,
                                      const int* __restrict__ blocks_in_use) {
  if (blocks_in_use) n_rows = min(n_rows, (long long)(*blocks_in_use) * 128);   // rows beyond the used blocks are never read
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = w; i < n_rows; i += n_warps) {
    const int rk = src_rank[i];
    if (rk < 0) {
      for (int c = lane * 8; c < width; c += 256)
        *reinterpret_cast<uint4*>(out + i * width + c) = make_uint4(0, 0, 0, 0);
      if (dot_out && lane == 0) dot_out[i] = 0.f;
      continue;
    }
    const __nv_bfloat16* s = reinterpret_cast<const __nv_bfloat16*>(src.p[rk]) + (long long)src_row[i] * src_ld;
    const float g = scale ? scale[i] : 1.f;
    float acc = 0.f;
    for (int c = lane * 8; c < width; c += 256) {
      uint4 v = *reinterpret_cast<const uint4*>(s + c);
      if (dot_with) {
        const uint4 d = *reinterpret_cast<const uint4*>(dot_with + i * width + c);
        const uint32_t a[4] = {v.x, v.y, v.z, v.w}, b[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 fa = unpack_bf16x2(a[e]), fb = unpack_bf16x2(b[e]);
          acc += fa.x * fb.x + fa.y * fb.y;
        }
      }
      if (scale) {
        uint32_t in[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = unpack_bf16x2(in[e]);
          in[e] = pack_bf16x2(f.x * g, f.y * g);
        }
        v = make_uint4(in[0], in[1], in[2], in[3]);
      }
      *reinterpret_cast<uint4*>(out + i * width + c) = v;
    }
    if (dot_out) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) dot_out[i] = acc;
    }
  }
}

// Deduplicated dispatch: a token with several slots on this rank crosses NVLink once.
// staging[r][row][:] = rank r's buffer[row][:] for every (r != self, row) with need[r*T + row] set.
__global__ void ep_stage_rows_kernel(PeerPtrs8 src, const unsigned char* __restrict__ need,
                                     __nv_bfloat16* __restrict__ staging, int world, int self, long long T,
                                     int width) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long items = (long long)world * T;
  for (long long i = w; i < items; i += n_warps) {
    const int r = (int)(i / T);
    if (r == self || !need[i]) continue;
    const long long row = i - (long long)r * T;
    const __nv_bfloat16* s = reinterpret_cast<const __nv_bfloat16*>(src.p[r]) + row * width;
    __nv_bfloat16* d = staging + i * width;
    // all loads of a batch are issued before the first store: up to 8 x 16 B per lane (4 KB per warp)
    // in flight over NVLink instead of one vector
    for (int c0 = lane * 8; c0 < width; c0 += 256 * 8) {
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (c0 + k * 256 < width) v[k] = *reinterpret_cast<const uint4*>(s + c0 + k * 256);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (c0 + k * 256 < width) *reinterpret_cast<uint4*>(d + c0 + k * 256) = v[k];
    }
  }
}

// Deduplicated combine: every expert rank first sums its slots of a token locally into
// partial[source rank][row]; the source then adds one partial row per contributing rank:
// y[row][:] += sum over r != self with sent[r*T + row] of rank r's partial[self*T + row][:].
__global__ void ep_reduce_rows_kernel(PeerPtrs8 part, const unsigned char* __restrict__ sent,
                                      __nv_bfloat16* __restrict__ y, int world, int self, long long T, int width) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = w; row < T; row += n_warps) {
    unsigned mask = 0;
    for (int r = 0; r < world; ++r)
      if (r != self && sent[(long long)r * T + row]) mask |= 1u << r;
    if (!mask) continue;
    for (int c = lane * 8; c < width; c += 256) {
      float acc[8];
      {
        const uint4 v = *reinterpret_cast<const uint4*>(y + row * width + c);
        const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), cc = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
        acc[0] = a.x; acc[1] = a.y; acc[2] = b.x; acc[3] = b.y; acc[4] = cc.x; acc[5] = cc.y; acc[6] = d.x; acc[7] = d.y;
      }
      // peer loads first (independent, all in flight together), sums afterwards
      uint4 pv[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < world && ((mask >> r) & 1u))
          pv[r] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(part.p[r]) +
                                                  ((long long)self * T + row) * width + c);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (!(r < world && ((mask >> r) & 1u))) continue;
        const uint4 v = pv[r];
        const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), cc = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
        acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y; acc[4] += cc.x; acc[5] += cc.y; acc[6] += d.x; acc[7] += d.y;
      }
      uint4 o;
      o.x = pack_bf16x2(acc[0], acc[1]);
      o.y = pack_bf16x2(acc[2], acc[3]);
      o.z = pack_bf16x2(acc[4], acc[5]);
      o.w = pack_bf16x2(acc[6], acc[7]);
      *reinterpret_cast<uint4*>(y + row * width + c) = o;
    }
  }
}

// dst_rank(i).buffer[dst_row(i), :] += weight(i) * rows[i, :]
__global__ void ep_scatter_add_kernel(PeerPtrs8 dst, const int* __restrict__ dst_rank,
                                      const int* __restrict__ dst_row, const float* __restrict__ weight,
                                      const __nv_bfloat16* __restrict__ rows, long long n_rows, int width,
                                      long long dst_ld) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = w; i < n_rows; i += n_warps) {
    if (dst_rank[i] < 0) continue;   // pad row of the expert-sorted layout
    const float g = weight ? weight[i] : 1.f;
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(dst.p[dst_rank[i]]) + (long long)dst_row[i] * dst_ld;
    for (int c = lane * 8; c < width; c += 256) {
      const uint4 v = *reinterpret_cast<const uint4*>(rows + i * width + c);
      const uint32_t in[4] = {v.x, v.y, v.z, v.w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack_bf16x2(in[e]);
        o[e] = pack_bf16x2(f.x * g, f.y * g);
      }
      asm volatile("red.relaxed.sys.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(d + c), "r"(o[0]),
                   "r"(o[1]), "r"(o[2]), "r"(o[3])
                   : "memory");
    }
  }
}

__global__ void peer_put_i32_kernel(int* __restrict__ dst, const int* __restrict__ src, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// Routing tables of every rank into one local array: dst[r * n + i] = peer r's src[i] (plain peer loads).
__global__ void ep_gather_tables_kernel(PeerPtrs8 src, int world, long long n, int* __restrict__ dst) {
  const long long total = (long long)world * n;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / n);
    dst[i] = reinterpret_cast<const int*>(src.p[r])[i - (long long)r * n];
  }
}

// Per-slot scalars back to the rank that routed the slot: peer src_rank[i] gets vals[i] at slot src_slot[i]
// (rows with src_rank < 0 are padding). Plain peer stores; the caller's barrier publishes them.
__global__ void ep_put_scalars_kernel(PeerPtrs8 dst, const int* __restrict__ src_rank, const int* __restrict__ src_slot,
                                      const float* __restrict__ vals, long long n, long long slots) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int r = src_rank[i], sl = src_slot[i];
    if (r < 0 || sl < 0 || sl >= slots) continue;
    reinterpret_cast<float*>(dst.p[r])[sl] = vals[i];
  }
}

int fill8(PeerPtrs8& d, const unsigned long long* s, int world) {
  if (world < 1 || world > 8) return -2;
  for (int i = 0; i < 8; ++i) d.p[i] = i < world ? s[i] : 0ull;
  return 0;
}
// out[C, R] = in[R, C]^T: 64 x 64 tiles through shared memory, both sides coalesced. ADD: out += (fp32).
// The adapter B of an expert stack is [N * r, E] as a parameter and [E, N * r] as a GEMM operand. Bound: HBM and, at these sizes,
// latency. 24576 / 32768 x 128: to bf16 8 us (strided copy and cast before: 23), to fp32 7 us (18).
constexpr int TR_T = 64;
template <typename Out, bool ADD>
__global__ void __launch_bounds__(256) transpose_kernel(const float* __restrict__ in, Out* __restrict__ out, long long R, long long C) {
  __shared__ float tile[TR_T][TR_T + 1];
  const unsigned tiles_c = (unsigned)((C + TR_T - 1) / TR_T);
  const long long r0 = (long long)(blockIdx.x / tiles_c) * TR_T, c0 = (long long)(blockIdx.x % tiles_c) * TR_T;
  const int x = threadIdx.x & 63, y0 = threadIdx.x >> 6;
  float v[TR_T / 4];
#pragma unroll
  for (int k = 0; k < TR_T / 4; ++k) {
    const int y = y0 + k * 4;
    v[k] = (r0 + y < R && c0 + x < C) ? in[(r0 + y) * C + c0 + x] : 0.f;
  }
#pragma unroll
  for (int k = 0; k < TR_T / 4; ++k) tile[y0 + k * 4][x] = v[k];
  __syncthreads();
#pragma unroll 4
  for (int k = 0; k < TR_T / 4; ++k) {
    const int y = y0 + k * 4;
    if (c0 + y >= C || r0 + x >= R) continue;
    Out* o = out + (c0 + y) * R + r0 + x;
    const float t = tile[x][y];
    if constexpr (ADD) *o += t;
    else if constexpr (sizeof(Out) == 2) *o = __float2bfloat16(t);
    else *o = t;
  }
}

}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

// q: [rows, cols/2] uint8, scale: [rows, cols/16] e4m3 bytes, pts: device fp32 scalar -> out [rows, cols] bf16
extern "C" int axb_nvfp4_dequant(const void* q, const void* scale, const float* pts, void* out, long long rows,
                                 long long cols, void* stream) {
  if (cols % 16) return -2;
  const long long nb = rows * (cols / 16);
  if (nb <= 0) return 0;
  int grid = (int)((nb / 2 + 255) / 256 > 148 * 16 ? 148 * 16 : (nb / 2 + 255) / 256);
  if (grid < 1) grid = 1;
  nvfp4_dequant_kernel<<<grid, 256, 0, ST(stream)>>>((const uint8_t*)q, (const uint8_t*)scale, pts,
                                                     (__nv_bfloat16*)out, nb, nb, nullptr);
  return (int)cudaGetLastError();
}

// batch of matrices (expert stacks): q [batch, rows, cols/2], scale [batch, rows, cols/16],
// pts [batch] fp32 -> out [batch, rows, cols] bf16, one launch. ``active`` (int32 [batch], optional):
// matrices whose entry is 0 are skipped and their output left untouched (experts without routed
// rows: what a decode step or a small batch saves).
extern "C" int axb_nvfp4_dequant_batched(const void* q, const void* scale, const float* pts, void* out,
                                         long long batch, long long rows, long long cols, const int* active,
                                         void* stream) {
  if (cols % 16) return -2;
  const long long per = rows * (cols / 16);
  const long long nb = batch * per;
  if (nb <= 0) return 0;
  int grid = (int)((nb / 2 + 255) / 256 > 148 * 16 ? 148 * 16 : (nb / 2 + 255) / 256);
  if (grid < 1) grid = 1;
  nvfp4_dequant_kernel<<<grid, 256, 0, ST(stream)>>>((const uint8_t*)q, (const uint8_t*)scale, pts,
                                                     (__nv_bfloat16*)out, nb, per, active);
  return (int)cudaGetLastError();
}

static int rows_grid(long long n_rows) {
  const long long want = (n_rows + 7) / 8;   // 8 warps (rows) per 256-thread block
  return (int)(want > 148 * 8 ? 148 * 8 : (want < 1 ? 1 : want));
}

// The pass table of axb_grouped_gemm_w4a16 for segments of counts[e] rows (device int64 [E]), each padded to whole 128-row blocks, one
// behind the other. passes int32 [max_blocks, 4], 16-byte aligned; n_pass [1]. Blocks from max_blocks on are left out.
extern "C" int axb_group_passes(const long long* counts, int E, int max_blocks, int* passes, int* n_pass, void* stream) {
  if (E < 1 || max_blocks < 0 || (reinterpret_cast<uintptr_t>(passes) & 15)) return -2;
  group_passes_kernel<<<1, RL_MAX_E, 0, ST(stream)>>>(counts, E, max_blocks, reinterpret_cast<int4*>(passes), n_pass);
  return (int)cudaGetLastError();
}

// Layout of a routed batch. expert [n] (n = T * k slots, expert ids), E <= 1024; slot_row [n], row_slot [max_blocks * 128] (slot of
// a padded row, -1 = pad), seg_start / seg_rows [E], blk_expert [max_blocks], n_blocks [1]; passes [max_blocks, 4], n_pass [1]: the
// passes of axb_grouped_gemm_w4a16 (first block, expert, rows in use, blocks), `passes` 16-byte aligned; scratch: ceil(n / 1024) * E
// ints. max_blocks >= ceil(n / 128) + E. A slot with an expert outside [0, E) has no row (slot_row -1) and sets *status.
extern "C" int axb_moe_route_layout(const long long* expert, int n, int E, int max_blocks, int* slot_row, int* row_slot,
                                    int* seg_start, int* seg_rows, int* blk_expert, int* n_blocks, int* passes, int* n_pass,
                                    int* scratch, int* status, void* stream) {
  if (reinterpret_cast<uintptr_t>(passes) & 15) return -2;
  if (E < 1 || E > RL_MAX_E || n < 0 || max_blocks < (n + 127) / 128 + E) return -2;
  cudaError_t e = cudaMemsetAsync(row_slot, 0xff, (size_t)max_blocks * 128 * sizeof(int), ST(stream));
  if (e != cudaSuccess) return (int)e;
  const int blocks = (n + RL_T - 1) / RL_T;
  if (blocks > 0) route_count_kernel<<<blocks, RL_T, E * (int)sizeof(int), ST(stream)>>>(expert, scratch, n, E);
  route_place_kernel<<<1, RL_MAX_E, 0, ST(stream)>>>(scratch, blocks, E, max_blocks, seg_start, seg_rows, blk_expert, n_blocks,
                                                     reinterpret_cast<int4*>(passes), n_pass);
  if (blocks > 0) {
    const int smem = 32 * E * (int)sizeof(unsigned short);      // at most 64 KB
    if (smem > 48 * 1024) {
      static std::atomic<unsigned long long> allowed{0};
      if (const int rc = axb_allow_smem((const void*)route_scatter_kernel, 64 * 1024, allowed)) return rc;
    }
    route_scatter_kernel<<<blocks, RL_T, smem, ST(stream)>>>(expert, scratch, slot_row, row_slot, n, E, status);
  }
  return (int)cudaGetLastError();
}

// out [n_rows, width] bf16, row_slot int32 [n_rows] (-1 = zero row), k slots per token, slot_scale fp32 [tokens * k] or NULL
extern "C" int axb_moe_dispatch_rows(const void* x, const int* row_slot, const float* slot_scale, void* out, long long n_rows,
                                     int width, int k, void* stream) {
  if (width % 8 || k < 1) return -2;
  if (n_rows <= 0) return 0;
  moe_dispatch_rows_kernel<<<rows_grid(n_rows), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)x, row_slot, slot_scale, (__nv_bfloat16*)out, n_rows, width, k);
  return (int)cudaGetLastError();
}

// out [n_tokens, width] = sum_j w[t, j] * ys[slot_row[t, j]]; w fp32 [n_tokens, k] or NULL (= 1)
extern "C" int axb_moe_combine_rows(const void* ys, const int* slot_row, const float* w, void* out,
                                    long long n_tokens, int k, int width, void* stream) {
  if (width % 8) return -2;
  if (n_tokens <= 0) return 0;
  moe_combine_rows_kernel<<<rows_grid(n_tokens * ((width + 255) / 256)), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)ys, slot_row, w, (__nv_bfloat16*)out, n_tokens, k, width);
  return (int)cudaGetLastError();
}

extern "C" int axb_moe_combine_dw(const void* dy, const void* ys, const int* slot_row, float* dw,
                                  long long n_slots, int k, int width, void* stream) {
  if (width % 8) return -2;
  if (n_slots <= 0) return 0;
  moe_combine_dw_kernel<<<rows_grid(n_slots), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)ys, slot_row, dw, n_slots, k, width);
  return (int)cudaGetLastError();
}

// src_rank[i] < 0 => zero row; scale (fp32 per row) / dot_with (bf16 [n_rows, width]) + dot_out are optional
extern "C" int axb_ep_gather_rows(const unsigned long long* src_ptrs, int world, const int* src_rank,
                                  const int* src_row, const float* scale, const void* dot_with, float* dot_out,
                                  void* out, long long n_rows, int width, long long src_ld, void* stream) {
  if (n_rows <= 0) return 0;
  if (width % 8 || src_ld % 8) return -2;
  PeerPtrs8 p;
  if (fill8(p, src_ptrs, world)) return -2;
  int grid = (int)((n_rows + 7) / 8 > 148 * 8 ? 148 * 8 : (n_rows + 7) / 8);
  ep_gather_rows_kernel<<<grid, 256, 0, ST(stream)>>>(p, src_rank, src_row, scale, (const __nv_bfloat16*)dot_with,
                                                      dot_out, (__nv_bfloat16*)out, n_rows, width, src_ld, nullptr);
  return (int)cudaGetLastError();
}
// the same over the first *blocks_in_use * 128 rows only (device-side count of the capacity-bounded plan)
extern "C" int axb_ep_gather_rows_n(const unsigned long long* src_ptrs, int world, const int* src_rank,
                                    const int* src_row, const float* scale, const void* dot_with, float* dot_out,
                                    void* out, long long n_rows, int width, long long src_ld, const int* blocks_in_use,
                                    void* stream) {
  if (n_rows <= 0) return 0;
  if (width % 8 || src_ld % 8) return -2;
  PeerPtrs8 p;
  if (fill8(p, src_ptrs, world)) return -2;
  int grid = (int)((n_rows + 7) / 8 > 148 * 8 ? 148 * 8 : (n_rows + 7) / 8);
  ep_gather_rows_kernel<<<grid, 256, 0, ST(stream)>>>(p, src_rank, src_row, scale, (const __nv_bfloat16*)dot_with,
                                                      dot_out, (__nv_bfloat16*)out, n_rows, width, src_ld, blocks_in_use);
  return (int)cudaGetLastError();
}

extern "C" int axb_ep_scatter_add(const unsigned long long* dst_ptrs, int world, const int* dst_rank,
                                  const int* dst_row, const float* weight, const void* rows, long long n_rows,
                                  int width, long long dst_ld, void* stream) {
  if (n_rows <= 0) return 0;
  if (width % 8 || dst_ld % 8) return -2;
  PeerPtrs8 p;
  if (fill8(p, dst_ptrs, world)) return -2;
  int grid = (int)((n_rows + 7) / 8 > 148 * 8 ? 148 * 8 : (n_rows + 7) / 8);
  ep_scatter_add_kernel<<<grid, 256, 0, ST(stream)>>>(p, dst_rank, dst_row, weight, (const __nv_bfloat16*)rows, n_rows,
                                                      width, dst_ld);
  return (int)cudaGetLastError();
}

extern "C" int axb_ep_stage_rows(const unsigned long long* src_ptrs, int world, int self, const void* need,
                                 void* staging, long long T, int width, void* stream) {
  if (T <= 0) return 0;
  if (width % 8) return -2;
  PeerPtrs8 p;
  if (fill8(p, src_ptrs, world)) return -2;
  const long long items = (long long)world * T;
  int grid = (int)((items + 7) / 8 > 148 * 8 ? 148 * 8 : (items + 7) / 8);
  ep_stage_rows_kernel<<<grid, 256, 0, ST(stream)>>>(p, (const unsigned char*)need, (__nv_bfloat16*)staging, world,
                                                     self, T, width);
  return (int)cudaGetLastError();
}

extern "C" int axb_ep_reduce_rows(const unsigned long long* part_ptrs, int world, int self, const void* sent,
                                  void* y, long long T, int width, void* stream) {
  if (T <= 0) return 0;
  if (width % 8) return -2;
  PeerPtrs8 p;
  if (fill8(p, part_ptrs, world)) return -2;
  int grid = (int)((T + 7) / 8 > 148 * 8 ? 148 * 8 : (T + 7) / 8);
  ep_reduce_rows_kernel<<<grid, 256, 0, ST(stream)>>>(p, (const unsigned char*)sent, (__nv_bfloat16*)y, world, self,
                                                      T, width);
  return (int)cudaGetLastError();
}

extern "C" int axb_ep_gather_tables(const unsigned long long* src_ptrs, int world, long long n, void* dst, void* stream) {
  PeerPtrs8 s;
  if (fill8(s, src_ptrs, world)) return -2;
  if (n <= 0) return 0;
  const long long total = (long long)world * n;
  int grid = (int)((total + 255) / 256 > 148 * 8 ? 148 * 8 : (total + 255) / 256);
  ep_gather_tables_kernel<<<grid, 256, 0, ST(stream)>>>(s, world, n, (int*)dst);
  return (int)cudaGetLastError();
}

extern "C" int axb_ep_put_scalars(const unsigned long long* dst_ptrs, int world, const void* src_rank,
                                  const void* src_slot, const void* vals, long long n, long long slots, void* stream) {
  PeerPtrs8 d;
  if (fill8(d, dst_ptrs, world)) return -2;
  if (n <= 0) return 0;
  int grid = (int)((n + 255) / 256 > 148 * 8 ? 148 * 8 : (n + 255) / 256);
  ep_put_scalars_kernel<<<grid, 256, 0, ST(stream)>>>(d, (const int*)src_rank, (const int*)src_slot, (const float*)vals, n, slots);
  return (int)cudaGetLastError();
}

extern "C" int axb_peer_put_i32(void* dst, const void* src, long long n, void* stream) {
  if (n <= 0) return 0;
  int grid = (int)((n + 255) / 256 > 148 * 4 ? 148 * 4 : (n + 255) / 256);
  peer_put_i32_kernel<<<grid, 256, 0, ST(stream)>>>((int*)dst, (const int*)src, n);
  return (int)cudaGetLastError();
}

// mode 0: bf16 out = in^T; 1: fp32 out += in^T; 2: fp32 out = in^T.  in fp32 [R, C], out [C, R], both dense.
extern "C" int axb_transpose(const float* in, void* out, long long R, long long C, int mode, void* stream) {
  if (R <= 0 || C <= 0) return 0;
  const long long tiles = ((R + TR_T - 1) / TR_T) * ((C + TR_T - 1) / TR_T);
  if (mode < 0 || mode > 2 || tiles > 0x7fffffffLL) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (mode == 0) transpose_kernel<__nv_bfloat16, false><<<(unsigned)tiles, 256, 0, st>>>(in, (__nv_bfloat16*)out, R, C);
  else if (mode == 1) transpose_kernel<float, true><<<(unsigned)tiles, 256, 0, st>>>(in, (float*)out, R, C);
  else transpose_kernel<float, false><<<(unsigned)tiles, 256, 0, st>>>(in, (float*)out, R, C);
  return (int)cudaGetLastError();
}
