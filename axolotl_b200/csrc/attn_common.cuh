// What the attention kernels of flash_varlen.cu and flash_wide.cu share: packed fp32 arithmetic, swizzle offsets, and the passes around
// the backward kernels (delta before, conversion of the fp32 dQ sums after).
#pragma once
#include "axb_common.cuh"

namespace {

AXB_DEVICE float fast_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two fp32 values in a register pair: one instruction each, rounded like the scalar ones
AXB_DEVICE uint64_t pack_b32x2(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
AXB_DEVICE uint64_t pack_f32x2(float a, float b) { return pack_b32x2(__float_as_uint(a), __float_as_uint(b)); }
AXB_DEVICE float2 unpack_f32x2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
AXB_DEVICE uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
AXB_DEVICE uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// byte offset of 8 consecutive bf16 (one 16-byte chunk) inside a [128 x 64] bf16 SW128 tile
AXB_DEVICE uint32_t sw128_chunk_off(int row, int chunk) {
  return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4);
}

// delta[h][t] = sum_d dO[t,h,d] * O[t,h,d]
// Bound: one read of dO and O. D / 8 threads of 16 bytes share a (token, head), a block covers TOK tokens x up to 8 heads so that
// its results leave as whole sectors of delta (one warp per (token, head) took 100 us for 7777 tokens x 64 heads of 64). 32 tokens
// while that gives every SM four blocks; below, a block of that size is a chain of up to 16 loads, and 8 tokens shorten it to 4
// (whole backward pass, heads of 128: 222 tokens, 3 heads 35.8 -> 27.6 us, 960 tokens, 32 heads 84 -> 65).
template <int D, int TOK>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ dout,
                                                         const __nv_bfloat16* __restrict__ out, float* __restrict__ delta,
                                                         long long T, int Hq, long long ld_do, long long ld_o) {
  constexpr int TPR = D / 8, ROWS = 256 / TPR;   // threads per (token, head), pairs per step
  constexpr int HEADS = 8;
  __shared__ float s[HEADS][TOK + 1];
  const long long t0 = (long long)blockIdx.x * TOK;
  const int h0 = blockIdx.y * HEADS, nh = min(HEADS, Hq - h0);
  const int sub = threadIdx.x % TPR, lane = threadIdx.x & 31, pairs = TOK * nh;
#pragma unroll 4
  for (int q0 = (int)(threadIdx.x >> 5) * (32 / TPR); q0 < pairs; q0 += ROWS) {     // the same for all lanes of a warp
    const int q = q0 + lane / TPR;                       // consecutive pairs: the heads of one token
    const int h = nh == HEADS ? q % HEADS : q % nh, tq = nh == HEADS ? q / HEADS : q / nh;
    const long long t = t0 + tq;
    float acc = 0.f;
    if (q < pairs && t < T) {
      const uint4 x = *reinterpret_cast<const uint4*>(dout + t * ld_do + (long long)(h0 + h) * D + sub * 8);
      const uint4 y = *reinterpret_cast<const uint4*>(out + t * ld_o + (long long)(h0 + h) * D + sub * 8);
      const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 u = unpack_bf16x2(xs[e]), v = unpack_bf16x2(ys[e]);
        acc += u.x * v.x + u.y * v.y;
      }
    }
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (sub == 0 && q < pairs) s[h][tq] = acc;
  }
  __syncthreads();
  const int h = threadIdx.x / TOK, t = threadIdx.x % TOK;
  if (h < nh && t0 + t < T) delta[(long long)(h0 + h) * T + t0 + t] = s[h][t];
}

template <int D>
void launch_attn_delta(const void* dout, const void* out, float* delta, long long T, int Hq, long long ld, cudaStream_t st) {
  const unsigned hb = (unsigned)((Hq + 7) / 8);
  const bool few = (T + 31) / 32 * hb < 4 * 148;
  const dim3 grid((unsigned)(few ? (T + 7) / 8 : (T + 31) / 32), hb);
  auto kern = few ? attn_delta_kernel<D, 8> : attn_delta_kernel<D, 32>;
  kern<<<grid, 256, 0, st>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)out, delta, T, Hq, ld, ld);
}

// What the backward passes move 16 bytes at a time, beyond what tensor maps check.
inline bool attn_bwd_aligned(const void* out, const void* dqkv, const void* dq_acc) {
  return ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dqkv) | reinterpret_cast<uintptr_t>(dq_acc)) & 15) == 0;
}

// Where the fp32 sum of dQ[row][col] stands (col = head * D + d, rows of `width`): four rows of a column side by side, so that a
// warp's 32 columns are 512 contiguous bytes of every group of four rows. The last rows % 4 rows are plain.
AXB_DEVICE long long dq_at(long long row, long long col, long long width, long long rows4) {
  return row < rows4 ? (row & ~3ll) * width + col * 4 + (row & 3) : row * width + col;
}

AXB_DEVICE void red_add_f32x4(float* to, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to), "f"(__uint_as_float(a)), "f"(__uint_as_float(b)),
               "f"(__uint_as_float(c)), "f"(__uint_as_float(d))
               : "memory");
}

AXB_DEVICE void red_add_f32x2(float* to, uint32_t a, uint32_t b) {
  asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(to), "f"(__uint_as_float(a)), "f"(__uint_as_float(b)) : "memory");
}
AXB_DEVICE void red_add_f32(float* to, uint32_t a) {
  asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(to), "f"(__uint_as_float(a)) : "memory");
}

// dq (bf16, q block of the fused gradient buffer) = dq_acc (fp32): a thread takes 8 columns of the four rows that lie side by side
__global__ void __launch_bounds__(256) dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dqkv, long long T, int width,
                                                         long long ld, int q_col0) {
  const int vecs = width / 8;
  const long long T4 = T & ~3ll, n = T4 / 4 * vecs + (T - T4) * vecs;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
    const long long t = v / vecs;
    const int c = (int)(v - t * vecs) * 8;
    if (t < T4 / 4) {
      const float4* src = reinterpret_cast<const float4*>(acc + t * 4 * width) + c;
      float4 f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = src[i];
      __nv_bfloat16* dst = dqkv + t * 4 * ld + q_col0 + c;
      *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(f[0].x, f[1].x), pack_bf16x2(f[2].x, f[3].x), pack_bf16x2(f[4].x, f[5].x), pack_bf16x2(f[6].x, f[7].x));
      *reinterpret_cast<uint4*>(dst + ld) = make_uint4(pack_bf16x2(f[0].y, f[1].y), pack_bf16x2(f[2].y, f[3].y), pack_bf16x2(f[4].y, f[5].y), pack_bf16x2(f[6].y, f[7].y));
      *reinterpret_cast<uint4*>(dst + 2 * ld) = make_uint4(pack_bf16x2(f[0].z, f[1].z), pack_bf16x2(f[2].z, f[3].z), pack_bf16x2(f[4].z, f[5].z), pack_bf16x2(f[6].z, f[7].z));
      *reinterpret_cast<uint4*>(dst + 3 * ld) = make_uint4(pack_bf16x2(f[0].w, f[1].w), pack_bf16x2(f[2].w, f[3].w), pack_bf16x2(f[4].w, f[5].w), pack_bf16x2(f[6].w, f[7].w));
    } else {
      const long long row = T4 + (t - T4 / 4);
      const float* src = acc + row * width + c;
      *reinterpret_cast<uint4*>(dqkv + row * ld + q_col0 + c) =
          make_uint4(pack_bf16x2(src[0], src[1]), pack_bf16x2(src[2], src[3]), pack_bf16x2(src[4], src[5]), pack_bf16x2(src[6], src[7]));
    }
  }
}

void launch_dq_convert(const float* acc, void* dqkv, long long T, int width, long long ld, int q_col0, cudaStream_t st) {
  const long long n = (T / 4 + T % 4) * (width / 8);
  const int grid = (int)((n + 255) / 256 > 148 * 16 ? 148 * 16 : (n + 255) / 256);
  dq_convert_kernel<<<grid, 256, 0, st>>>(acc, (__nv_bfloat16*)dqkv, T, width, ld, q_col0);
}

}  // namespace
