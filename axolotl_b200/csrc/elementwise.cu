// Memory-bound fused ops for sm_100a: RMSNorm (+residual add) fwd/bwd, RoPE (+optional per-head
// q/k RMSNorm for Qwen3) fwd/bwd, SwiGLU / GeGLU fwd/bwd, embedding gather / scatter-add,
// in-place cross-entropy fwd+bwd over a logits chunk, fused multi-tensor AdamW with global-norm
// clipping. All kernels move 16-byte vectors and keep statistics in fp32.
//
// These replace the reference's Triton kernels (src/axolotl/kernels/swiglu.py, geglu.py,
// gemma4_fused_rope.py), the HF eager RMSNorm / rotary chains and torch's fused AdamW.
#include "axb_common.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int NT>
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.f;
  if (w == 0) {
    r = warp_sum(r);
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}
template <int NT>
__device__ __forceinline__ float block_max(float v, float* sh) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : -INFINITY;
  if (w == 0) {
    r = warp_max(r);
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}

struct bf16x8 {
  uint4 u;
};
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z),
         d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8]) {
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 packed8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]);
  u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]);
  u.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ---------------------------------------------------------------------------------- RMSNorm
// h = x (+ res);  res_out = h (optional);  y = h * rstd * (w + w_offset)
// Bound: HBM. A thread owns NV 16-byte vectors of a row (NV = 0: any number, in a loop), all requested before the first is
// used, and keeps them packed while the row is summed: 8192 x 4096 with a residual 60 -> 49 us (4 x 67 MB, L2 flushed).
constexpr int NORM_T = 256;
template <int NV>
__global__ void __launch_bounds__(NORM_T)
    rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                       const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                       __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out, int H,
                       float eps, float w_offset) {
  __shared__ float sh[32];
  pdl_launch_dependents();
  pdl_wait();
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * H;
  const __nv_bfloat16* rr = res ? res + row * H : nullptr;
  float ss = 0.f;
  auto add = [&](uint4 a, uint4 b, float (&f)[8]) {        // x (+ res)
    unpack8(a, f);
    if (rr) {
      float g[8];
      unpack8(b, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
    }
  };
  if constexpr (NV > 0) {
    uint4 a[NV], b[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = (k * NORM_T + threadIdx.x) * 8;
      a[k] = b[k] = make_uint4(0, 0, 0, 0);
      if (i < H) {
        a[k] = *reinterpret_cast<const uint4*>(xr + i);
        if (rr) b[k] = *reinterpret_cast<const uint4*>(rr + i);
      }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = (k * NORM_T + threadIdx.x) * 8;
      float f[8];
      add(a[k], b[k], f);
      if (res_out) {
        // the residual stream is rounded to bf16 first so that forward and backward see the same h
        a[k] = packed8(f);
        if (i < H) *reinterpret_cast<uint4*>(res_out + row * H + i) = a[k];
        unpack8(a[k], f);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
    ss = block_sum<NORM_T>(ss, sh);
    const float rstd = rsqrtf(ss / H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = (k * NORM_T + threadIdx.x) * 8;
      if (i >= H) continue;
      float f[8], wv[8];
      if (res_out) unpack8(a[k], f);
      else add(a[k], b[k], f);
      load8(w + i, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * (wv[j] + w_offset);
      store8(y + row * H + i, f);
    }
  } else {
    for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8) {
      float f[8];
      add(*reinterpret_cast<const uint4*>(xr + i), rr ? *reinterpret_cast<const uint4*>(rr + i) : make_uint4(0, 0, 0, 0), f);
      if (res_out) {
        const uint4 u = packed8(f);
        *reinterpret_cast<uint4*>(res_out + row * H + i) = u;
        unpack8(u, f);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
    }
    ss = block_sum<NORM_T>(ss, sh);
    const float rstd = rsqrtf(ss / H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
    for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8) {
      float f[8], wv[8];
      if (res_out) load8(res_out + row * H + i, f);
      else add(*reinterpret_cast<const uint4*>(xr + i), rr ? *reinterpret_cast<const uint4*>(rr + i) : make_uint4(0, 0, 0, 0), f);
      load8(w + i, wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * (wv[j] + w_offset);
      store8(y + row * H + i, f);
    }
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres). Each thread owns fixed columns, so the
// weight gradient is accumulated in registers over the rows of the block and flushed once.
// Bound: HBM. The blocks stay resident and walk over rows; the three inputs of the next row are requested before the
// present row's reduction, so that a block always has loads in flight, and the row is read once (packed in registers). The
// flush goes through shared memory, whole 128-byte lines per warp: the strided atomics of eight blocks per SM cost more
// than the pass itself. 8192 x 4096 83 -> 54 us; 4096 x 2048 with a weight gradient 115 -> 28 us (L2 flushed).
template <int NV, bool DW>
__global__ void __launch_bounds__(NORM_T)
    rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                       const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                       float* __restrict__ dw, int H, int rows, float w_offset) {
  __shared__ float sh[2][NORM_T / 32];
  __shared__ float s_dw[DW ? NORM_T * 8 : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float dw_acc[DW ? NV : 1][8];
  if (DW) {
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) dw_acc[k][j] = 0.f;
  }
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wv[NV], a[NV], b[NV], d[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (k * NORM_T + threadIdx.x) * 8;
    wv[k] = i < H ? *reinterpret_cast<const uint4*>(w + i) : zero;
  }
  float rstd = 0.f;
  auto fetch = [&](long long row) {
    rstd = rstd_in[row];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = (k * NORM_T + threadIdx.x) * 8;
      a[k] = b[k] = d[k] = zero;
      if (i < H) {
        a[k] = *reinterpret_cast<const uint4*>(dy + row * H + i);
        b[k] = *reinterpret_cast<const uint4*>(h + row * H + i);
        if (dres) d[k] = *reinterpret_cast<const uint4*>(dres + row * H + i);
      }
    }
  };
  long long row = blockIdx.x;
  if (row < rows) fetch(row);
  int turn = 0;
  for (; row < rows; row += gridDim.x, turn ^= 1) {
    uint4 ca[NV], cb[NV], cd[NV];
    const float rs = rstd;
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      ca[k] = a[k];
      cb[k] = b[k];
      cd[k] = d[k];
      float fa[8], fb[8], fw[8];
      unpack8(ca[k], fa);
      unpack8(cb[k], fb);
      unpack8(wv[k], fw);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += fa[j] * (fw[j] + w_offset) * fb[j] * rs;
    }
    if (row + gridDim.x < rows) fetch(row + gridDim.x);
    dot = warp_sum(dot);
    if (lane == 0) sh[turn][warp] = dot;        // two slots in turn: one barrier per row
    __syncthreads();
    dot = 0.f;
#pragma unroll
    for (int q = 0; q < NORM_T / 32; ++q) dot += sh[turn][q];
    dot /= H;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = (k * NORM_T + threadIdx.x) * 8;
      if (i >= H) continue;
      float fa[8], fb[8], fw[8], o[8];
      unpack8(ca[k], fa);
      unpack8(cb[k], fb);
      unpack8(wv[k], fw);
      unpack8(cd[k], o);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = fb[j] * rs;
        const float g = rs * (fa[j] * (fw[j] + w_offset) - xhat * dot);
        if (DW) dw_acc[k][j] += fa[j] * xhat;
        o[j] = dres ? o[j] + g : g;
      }
      store8(dx + row * H + i, o);
    }
  }
  if constexpr (DW) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) s_dw[threadIdx.x * 8 + j] = dw_acc[k][j];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = k * NORM_T * 8 + j * NORM_T + threadIdx.x;
        if (i < H) atomicAdd(dw + i, s_dw[j * NORM_T + threadIdx.x]);
      }
    }
  }
}
// rows wider than 4 x 2048 elements: the first four vectors of a thread accumulate their weight gradient in registers
__global__ void __launch_bounds__(NORM_T)
    rmsnorm_bwd_wide_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in,
                       const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                       float* __restrict__ dw, int H, int rows, float w_offset) {
  __shared__ float sh[32];
  float dw_acc[4][8];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[a][j] = 0.f;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float dot = 0.f;
    for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8) {
      float a[8], b[8], c[8];
      load8(dy + row * H + i, a);
      load8(h + row * H + i, b);
      load8(w + i, c);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += a[j] * (c[j] + w_offset) * b[j] * rstd;
    }
    dot = block_sum<NORM_T>(dot, sh) / H;
    int k = 0;
    for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8, ++k) {
      float a[8], b[8], c[8], o[8];
      load8(dy + row * H + i, a);
      load8(h + row * H + i, b);
      load8(w + i, c);
      if (dres) load8(dres + row * H + i, o);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = b[j] * rstd;
        const float g = rstd * (a[j] * (c[j] + w_offset) - xhat * dot);
        if (dw) {
          if (k < 4) dw_acc[k][j] += a[j] * xhat;
          else atomicAdd(dw + i + j, a[j] * xhat);
        }
        o[j] = dres ? o[j] + g : g;
      }
      store8(dx + row * H + i, o);
    }
  }
  if (dw) {
    int k = 0;
    for (int i = threadIdx.x * 8; i < H && k < 4; i += NORM_T * 8, ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dw + i + j, dw_acc[k][j]);
  }
}

// ---------------------------------------------------------------------------------- RoPE
// Rotates the q and k heads of a fused [T, (Hq + 2*Hk) * D] projection in place (rotate-half
// convention: out = x*cos + rotate_half(x)*sin, angles = pos * inv_freq[i], i < D/2).
// With norm weights given, a per-head RMSNorm over D is applied first (Qwen3 q_norm / k_norm),
// and the per-head rstd is saved for the backward pass. sign = -1 gives the inverse rotation.
__global__ void rope_qk_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ pos,
                               const float* __restrict__ inv_freq, int T, int Hq, int Hk, int D,
                               long long row_stride, float sign, float attn_scale,
                               const __nv_bfloat16* __restrict__ qn_w,
                               const __nv_bfloat16* __restrict__ kn_w, float* __restrict__ rstd_out,
                               float eps) {
  // one warp per (token, head); lane handles pairs (i, i + D/2)
  const int warps_per_block = blockDim.x >> 5;
  const long long gw = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int nh = Hq + Hk;
  if (gw >= (long long)T * nh) return;
  const int t = (int)(gw / nh);
  const int hd = (int)(gw % nh);
  __nv_bfloat16* p = qkv + (long long)t * row_stride + (long long)hd * D;
  const float ps = (float)pos[t];
  const int half = D >> 1;
  const __nv_bfloat16* nw = (hd < Hq) ? qn_w : kn_w;
  float rstd = 1.f;
  if (nw) {
    float ss = 0.f;
    for (int i = lane; i < D; i += 32) {
      float v = __bfloat162float(p[i]);
      ss += v * v;
    }
    ss = warp_sum(ss);
    rstd = rsqrtf(ss / D + eps);
    if (lane == 0 && rstd_out) rstd_out[gw] = rstd;
  }
  for (int i = lane; i < half; i += 32) {
    float s, c;
    sincosf(ps * inv_freq[i], &s, &c);
    s *= sign * attn_scale;
    c *= attn_scale;
    float a = __bfloat162float(p[i]);
    float b = __bfloat162float(p[i + half]);
    if (nw) {
      a = __bfloat162float(__float2bfloat16(a * rstd * __bfloat162float(nw[i])));
      b = __bfloat162float(__float2bfloat16(b * rstd * __bfloat162float(nw[i + half])));
    }
    p[i] = __float2bfloat16(a * c - b * s);
    p[i + half] = __float2bfloat16(b * c + a * s);
  }
}

// Fast path without q/k norm: one warp per (token, group of heads). Each lane computes the sine / cosine of its two
// angles ONCE and reuses them for the group's heads (the angles depend on the position
// only), and moves bf16 pairs (4-byte accesses, 128 B per warp instruction). sign = -1 is the
// inverse rotation, i.e. the backward pass.
// Bound: latency for short batches, HBM for long ones. Four heads are loaded before the first is stored (in place, the
// compiler cannot move a load above an earlier store), and heads are spread over blockIdx.y while there are few tokens:
// 960 rows of 40 heads 15.6 -> 5.7 us, 8192 rows 38 -> 32 us (one warp walking all heads of a row, one head at a time, before).
// `rot` <= D: only the first `rot` dimensions of a head rotate (partial rotary embeddings: pairs (j, j + rot / 2));
// the rest of the head passes through untouched.
constexpr int ROPE_H = 4;
__global__ void rope_fast_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ pos,
                                 const float* __restrict__ inv_freq, int T, int nh, int D,
                                 long long row_stride, float sign, float attn_scale, int rot) {
  const int warps_per_block = blockDim.x >> 5;
  const long long t = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  const int half = rot >> 1;
  const float ps = (float)pos[t];
  __nv_bfloat16* row = qkv + t * row_stride;
  const int groups = (nh + ROPE_H - 1) / ROPE_H;
  for (int j = 2 * lane; j < half; j += 64) {
    float s0, c0, s1, c1;
    sincosf(ps * inv_freq[j], &s0, &c0);
    sincosf(ps * inv_freq[j + 1], &s1, &c1);
    s0 *= sign * attn_scale;
    s1 *= sign * attn_scale;
    c0 *= attn_scale;
    c1 *= attn_scale;
    for (int g = blockIdx.y; g < groups; g += gridDim.y) {
      uint32_t* p0 = reinterpret_cast<uint32_t*>(row + (long long)g * ROPE_H * D + j);
      uint32_t ua[ROPE_H], ub[ROPE_H];
#pragma unroll
      for (int h = 0; h < ROPE_H; ++h) {
        if (g * ROPE_H + h >= nh) break;
        ua[h] = p0[(h * D) >> 1];
        ub[h] = p0[(h * D + half) >> 1];
      }
#pragma unroll
      for (int h = 0; h < ROPE_H; ++h) {
        if (g * ROPE_H + h >= nh) break;
        const float2 a = unpack_bf16x2(ua[h]), b = unpack_bf16x2(ub[h]);
        p0[(h * D) >> 1] = pack_bf16x2(a.x * c0 - b.x * s0, a.y * c1 - b.y * s1);
        p0[(h * D + half) >> 1] = pack_bf16x2(b.x * c0 + a.x * s0, b.y * c1 + a.y * s1);
      }
    }
  }
}
// eight blocks per SM, but never more head groups than there are
static dim3 rope_grid(int T, int nh) {
  const int bx = (T + 7) / 8, groups = (nh + ROPE_H - 1) / ROPE_H;
  int by = (148 * 8 + bx - 1) / bx;
  if (by > groups) by = groups;
  return dim3((unsigned)bx, (unsigned)(by < 1 ? 1 : by));
}

// Backward of (per-head RMSNorm ->) RoPE for the fused q/k gradient buffer, in place.
// x_pre holds the pre-norm projection (needed only when norm weights are given).
// NMAX: rotation pairs a lane keeps in registers (D <= 64 * NMAX).
template <int NMAX>
__global__ void rope_qk_bwd_kernel(__nv_bfloat16* __restrict__ dqkv,
                                   const __nv_bfloat16* __restrict__ x_pre,
                                   const int* __restrict__ pos, const float* __restrict__ inv_freq,
                                   int T, int Hq, int Hk, int D, long long row_stride,
                                   long long x_row_stride, float attn_scale,
                                   const __nv_bfloat16* __restrict__ qn_w,
                                   const __nv_bfloat16* __restrict__ kn_w,
                                   const float* __restrict__ rstd_in, float* __restrict__ dqn_w,
                                   float* __restrict__ dkn_w) {
  const int warps_per_block = blockDim.x >> 5;
  const long long gw = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int nh = Hq + Hk;
  if (gw >= (long long)T * nh) return;
  const int t = (int)(gw / nh);
  const int hd = (int)(gw % nh);
  __nv_bfloat16* g = dqkv + (long long)t * row_stride + (long long)hd * D;
  const float ps = (float)pos[t];
  const int half = D >> 1;
  const __nv_bfloat16* nw = (hd < Hq) ? qn_w : kn_w;
  float* dnw = (hd < Hq) ? dqn_w : dkn_w;
  // inverse rotation first
  float ga[NMAX], gb[NMAX];
  int n = 0;
  for (int i = lane; i < half; i += 32, ++n) {
    float s, c;
    sincosf(ps * inv_freq[i], &s, &c);
    s *= attn_scale;
    c *= attn_scale;
    const float a = __bfloat162float(g[i]);
    const float b = __bfloat162float(g[i + half]);
    ga[n] = a * c + b * s;
    gb[n] = b * c - a * s;
  }
  if (!nw) {
    n = 0;
    for (int i = lane; i < half; i += 32, ++n) {
      g[i] = __float2bfloat16(ga[n]);
      g[i + half] = __float2bfloat16(gb[n]);
    }
    return;
  }
  const __nv_bfloat16* x = x_pre + (long long)t * x_row_stride + (long long)hd * D;
  const float rstd = rstd_in[gw];
  float dot = 0.f;
  n = 0;
  for (int i = lane; i < half; i += 32, ++n) {
    const float xa = __bfloat162float(x[i]) * rstd, xb = __bfloat162float(x[i + half]) * rstd;
    const float wa = __bfloat162float(nw[i]), wb = __bfloat162float(nw[i + half]);
    dot += ga[n] * wa * xa + gb[n] * wb * xb;
    if (dnw) {
      atomicAdd(dnw + i, ga[n] * xa);
      atomicAdd(dnw + i + half, gb[n] * xb);
    }
  }
  dot = warp_sum(dot) / D;
  n = 0;
  for (int i = lane; i < half; i += 32, ++n) {
    const float xa = __bfloat162float(x[i]) * rstd, xb = __bfloat162float(x[i + half]) * rstd;
    const float wa = __bfloat162float(nw[i]), wb = __bfloat162float(nw[i + half]);
    g[i] = __float2bfloat16(rstd * (ga[n] * wa - xa * dot));
    g[i + half] = __float2bfloat16(rstd * (gb[n] * wb - xb * dot));
  }
}

// ---------------------------------------------------------------------------------- GLU
// Special-function-unit forms (ex2 / rcp / tanh approximations, a couple of ulp: far below the bf16
// rounding of the results); an IEEE division per element would make these kernels instruction-bound.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sigmoid_fast(float g) { return __fdividef(1.f, 1.f + __expf(-g)); }
// kind 0: silu, 1: gelu (tanh form), 2: g * sigmoid(1.702 g), whose GLU multiplies by (up + 1) (gpt-oss experts)
__device__ __forceinline__ float act_fwd(float g, int kind) {
  if (kind == 0) return g * sigmoid_fast(g);  // silu
  if (kind == 2) return g * sigmoid_fast(1.702f * g);
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;  // gelu tanh
  const float t = tanh_fast(k0 * (g + k1 * g * g * g));
  return 0.5f * g * (1.f + t);
}
__device__ __forceinline__ float act_bwd(float g, int kind) {
  if (kind == 0) {
    const float s = sigmoid_fast(g);
    return s * (1.f + g * (1.f - s));
  }
  if (kind == 2) {
    const float s = sigmoid_fast(1.702f * g);
    return s * (1.f + 1.702f * g * (1.f - s));
  }
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float t = tanh_fast(k0 * (g + k1 * g * g * g));
  return 0.5f * (1.f + t) + 0.5f * g * (1.f - t * t) * k0 * (1.f + 3.f * k1 * g * g);
}
// gu: [T, 2I] (gate | up);  h: [T, I] = act(gate) * up. With limit > 0 (clamped SwiGLU of the
// DeepSeek-V4 / gpt-oss experts): act(min(gate, limit)) * clamp(up, -limit, limit), and the
// gradients vanish where the clamp is active.
// `blocks_in_use` (optional, device): only the first *blocks_in_use * 128 rows are processed: the padded expert layout
// of a capacity-bounded plan uses a data-dependent prefix of its row buffer and nothing reads the rest.
__global__ void glu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ h,
                               long long T, int I, int kind, float limit, const int* __restrict__ blocks_in_use) {
  if (blocks_in_use) T = min(T, (long long)(*blocks_in_use) * 128);
  const long long nvec = T * (I / 8);
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec;
       v += (long long)gridDim.x * blockDim.x) {
    const long long t = v / (I / 8);
    const int c = (int)(v % (I / 8)) * 8;
    float g[8], u[8], o[8];
    load8(gu + t * 2 * I + c, g);
    load8(gu + t * 2 * I + I + c, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gc = limit > 0.f ? fminf(g[j], limit) : g[j];
      const float uc = limit > 0.f ? fminf(fmaxf(u[j], -limit), limit) : u[j];
      o[j] = act_fwd(gc, kind) * (kind == 2 ? uc + 1.f : uc);
    }
    store8(h + t * I + c, o);
  }
}
// dgu[T,2I]: d_gate = dh * up * act'(gate), d_up = dh * act(gate). dgu may alias gu.
__global__ void glu_bwd_kernel(const __nv_bfloat16* __restrict__ dh,
                               const __nv_bfloat16* __restrict__ gu,
                               __nv_bfloat16* __restrict__ dgu, long long T, int I, int kind,
                               float limit, const int* __restrict__ blocks_in_use) {
  if (blocks_in_use) T = min(T, (long long)(*blocks_in_use) * 128);
  const long long nvec = T * (I / 8);
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec;
       v += (long long)gridDim.x * blockDim.x) {
    const long long t = v / (I / 8);
    const int c = (int)(v % (I / 8)) * 8;
    float g[8], u[8], d[8], og[8], ou[8];
    load8(gu + t * 2 * I + c, g);
    load8(gu + t * 2 * I + I + c, u);
    load8(dh + t * I + c, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const bool g_in = !(limit > 0.f) || g[j] <= limit;
      const bool u_in = !(limit > 0.f) || (u[j] >= -limit && u[j] <= limit);
      const float gc = g_in ? g[j] : limit;
      const float uc = u_in ? u[j] : (u[j] > 0.f ? limit : -limit);
      og[j] = g_in ? d[j] * (kind == 2 ? uc + 1.f : uc) * act_bwd(gc, kind) : 0.f;
      ou[j] = u_in ? d[j] * act_fwd(gc, kind) : 0.f;
    }
    store8(dgu + t * 2 * I + c, og);
    store8(dgu + t * 2 * I + I + c, ou);
  }
}

// ---------------------------------------------------------------------------------- DoRA weight norm
// norm[n] = sqrt(max(w2[n] + 2 s <W, BA>_n + s^2 |BA|_n^2, tiny)) with <W, BA>_n = sum_r WA[n,r] B[n,r] and
// |BA|_n^2 = sum_{q,r} B[n,q] G[q,r] B[n,r], G = A A^T [R, R] (fp32). One thread per output row, G in shared
// memory: the row-wise tail of the reference's fused DoRA-norm kernel (src/axolotl/kernels/dora.py:16-147)
// after the skinny tcgen05 GEMM W A^T.
__global__ void dora_norm_kernel(const float* __restrict__ WA, const float* __restrict__ B, const float* __restrict__ G,
                                 const float* __restrict__ w2, float* __restrict__ norm, long long N, int R, float s) {
  extern __shared__ float sG[];
  for (int i = threadIdx.x; i < R * R; i += blockDim.x) sG[i] = G[i];
  __syncthreads();
  const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const float* b = B + n * R;
  const float* wa = WA + n * R;
  float cross = 0.f, quad = 0.f;
  for (int r = 0; r < R; ++r) {
    const float br = b[r];
    cross += wa[r] * br;
    float acc = 0.f;
    for (int q = 0; q < R; ++q) acc += b[q] * sG[q * R + r];
    quad += acc * br;
  }
  norm[n] = sqrtf(fmaxf(w2[n] + 2.f * s * cross + s * s * quad, 1e-12f));
}

// ---------------------------------------------------------------------------------- embedding
__global__ void embedding_fwd_kernel(const __nv_bfloat16* __restrict__ table,
                                     const long long* __restrict__ ids,
                                     __nv_bfloat16* __restrict__ out, long long T, int H,
                                     long long vocab) {
  const long long nvec = T * (H / 8);
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec;
       v += (long long)gridDim.x * blockDim.x) {
    const long long t = v / (H / 8);
    const int c = (int)(v % (H / 8)) * 8;
    long long id = ids[t];
    if (c == 0) (void)AXB_INDEX_OK(AXB_SITE_EMBED_ID, id, vocab);
    if (id < 0 || id >= vocab) id = 0;
    *reinterpret_cast<uint4*>(out + t * H + c) =
        *reinterpret_cast<const uint4*>(table + id * H + c);
  }
}
// One thread per VEC elements of a row. VEC = 8: one 16-byte load and two 16-byte reductions (4096 rows of 2048: 29 -> 17 us
// with one element and one reduction per thread before); VEC = 1 for rows or tables off the 16-byte grid.
template <int VEC>
__global__ void embedding_bwd_kernel(const __nv_bfloat16* __restrict__ dout,
                                     const long long* __restrict__ ids, float* __restrict__ dtable,
                                     long long T, int H, long long vocab) {
  const int per = H / VEC;
  const long long n = T * per;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / per;
    const int c = (int)(i % per) * VEC;
    const long long id = ids[t];
    if (c == 0) (void)AXB_INDEX_OK(AXB_SITE_EMBED_GRAD_ID, id, vocab);
    if (id < 0 || id >= vocab) continue;
    float* dst = dtable + id * H + c;
    if constexpr (VEC == 8) {
      float f[8];
      load8(dout + t * H + c, f);
      atomicAdd(reinterpret_cast<float4*>(dst), make_float4(f[0], f[1], f[2], f[3]));
      atomicAdd(reinterpret_cast<float4*>(dst + 4), make_float4(f[4], f[5], f[6], f[7]));
    } else {
      atomicAdd(dst, __bfloat162float(dout[t * H + c]));
    }
  }
}

// ---------------------------------------------------------------------------------- cross entropy
// One block per row of a [R, V] bf16 logits chunk (optionally soft-capped). Computes
//   loss[r] = logsumexp(z) - z[label]   (0 when label == ignore_index)
// and overwrites the row with d loss_total / d z = (softmax(z) - onehot) * grad_scale, so the
// caller can feed the buffer straight into the dX / dW GEMMs. lse[r] is also returned.
// Bound: HBM for one read and one write of the row; the second read comes from L2, where three blocks of 512 threads per SM leave
// room for it (four did not, and a separate pass for the maximum read the row a third time). The maximum and the sum run
// together, rebased once per CE_U vectors of a thread, which are loaded together. 2048 rows of 128256: 300 -> 231 us
// (4.5 TB/s of read + write), 959 rows 159 -> 118. Narrow rows want smaller blocks (2048 rows of 8192: 512 threads 34 us,
// 256 threads 24, before 28; of 32000: 65 / 62 / 68; of 50257: 97 / 100 / 103).
constexpr int CE_U = 4, CE_NARROW = 40960;
constexpr int ENT_T = 512;   // entropy kernel below
// CAP: the logits are soft-capped first, z' = cap * tanh(z / cap) (Gemma 2 final_logit_softcapping); the
// gradient written back is with respect to the raw z.
template <bool CAP, int NT>
__global__ void __launch_bounds__(NT, 1536 / NT)
    ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
                      float* __restrict__ loss, float* __restrict__ lse_out, int V,
                      long long ld, float grad_scale, long long ignore_index, int write_grad, float cap) {
  const float inv_cap = CAP ? 1.f / cap : 0.f;
  auto eff = [&](float v) -> float {
    if constexpr (CAP) return cap * tanhf(v * inv_cap);
    else return v;
  };
  __shared__ float sh[32];
  const long long r = blockIdx.x;
  __nv_bfloat16* z = logits + r * ld;
  const long long label = labels[r];
  if (threadIdx.x == 0 && label != ignore_index) (void)AXB_INDEX_OK(AXB_SITE_CE_LABEL, label, V);
  const bool ignored = (label == ignore_index) || label < 0 || label >= V;
  if (ignored && !lse_out) {
    if (threadIdx.x == 0) loss[r] = 0.f;
    if (write_grad) {
      const uint4 zero = make_uint4(0, 0, 0, 0);
      const int v8 = V & ~7;
      for (int i = threadIdx.x * 8; i < v8; i += NT * 8)
        *reinterpret_cast<uint4*>(z + i) = zero;
      for (int i = v8 + threadIdx.x; i < V; i += NT) z[i] = __float2bfloat16(0.f);
    }
    return;
  }
  const int nvec = V >> 3, ti = (nvec << 3) + (int)threadIdx.x;   // the V % 8 elements behind the last vector: one thread each
  const uint4* zv = reinterpret_cast<const uint4*>(z);
  // CE_U vectors of a thread, the first at v; a vector past the end is all -inf
  auto load = [&](int v, uint4 (&u)[CE_U]) {
#pragma unroll
    for (int k = 0; k < CE_U; ++k)
      u[k] = v + k * NT < nvec ? zv[v + k * NT] : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);
  };
  float mx = -INFINITY, se = 0.f;               // running maximum and sum relative to it
  auto rebase = [&](float m) -> float {         // -inf has no distance to itself: a base of 0 leaves its exp 0
    const float nm = fmaxf(mx, m), b = nm == -INFINITY ? 0.f : nm;
    se *= __expf(mx - b);
    mx = nm;
    return b;
  };
  for (int v = threadIdx.x; v < nvec; v += CE_U * NT) {
    uint4 u[CE_U];
    load(v, u);
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < CE_U; ++k) {
      float f[8];
      unpack8(u[k], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, f[j]);   // tanh is increasing: only the maximum is capped
    }
    const float b = rebase(eff(m));             // capped, a group of -inf is a group of -cap: finite terms like all others
    float part = 0.f;                           // summed on its own: a long row loses less
#pragma unroll
    for (int k = 0; k < CE_U; ++k) {
      if (CAP && v + k * NT >= nvec) continue;        // capped, -inf would count
      float f[8];
      unpack8(u[k], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) part += __expf(eff(f[j]) - b);
    }
    se += part;
  }
  const float zt = ti < V ? eff(__bfloat162float(z[ti])) : 0.f;
  if (ti < V) {
    const float b = rebase(zt);
    se += __expf(zt - b);
  }
  const float m_all = block_max<NT>(mx, sh);
  se = block_sum<NT>(se * __expf(mx - m_all), sh);
  const float lse = m_all + logf(se);
  if (threadIdx.x == 0) {
    if (lse_out) lse_out[r] = lse;
    loss[r] = ignored ? 0.f : lse - eff(__bfloat162float(z[label]));
  }
  if (!write_grad) return;
  __syncthreads();
  const float gs = ignored ? 0.f : grad_scale;
  auto grad = [&](float ze, bool hit) -> float {
    float pr = __expf(ze - lse);
    if (hit) pr -= 1.f;
    if constexpr (CAP) pr *= 1.f - (ze * inv_cap) * (ze * inv_cap);   // d z' / d z = 1 - tanh^2
    return pr * gs;
  };
  for (int v = threadIdx.x; v < nvec; v += CE_U * NT) {
    uint4 u[CE_U];
    load(v, u);
#pragma unroll
    for (int k = 0; k < CE_U; ++k) {
      const int vk = v + k * NT;
      if (vk >= nvec) break;
      const int hit = (label >> 3) == vk ? (int)(label & 7) : -1;
      float f[8];
      unpack8(u[k], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = grad(eff(f[j]), j == hit);
      store8(z + vk * 8LL, f);
    }
  }
  if (ti < V) z[ti] = __float2bfloat16(grad(zt, ti == label));
}
template <bool CAP>
static int ce_launch(void* logits, const long long* labels, float* loss, float* lse, long long rows, int V, long long ld,
                     float grad_scale, long long ignore_index, int write_grad, float cap, cudaStream_t st) {
  __nv_bfloat16* z = (__nv_bfloat16*)logits;
  if (V <= CE_NARROW)
    ce_fwd_bwd_kernel<CAP, 256><<<(unsigned)rows, 256, 0, st>>>(z, labels, loss, lse, V, ld, grad_scale, ignore_index, write_grad, cap);
  else
    ce_fwd_bwd_kernel<CAP, 512><<<(unsigned)rows, 512, 0, st>>>(z, labels, loss, lse, V, ld, grad_scale, ignore_index, write_grad, cap);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------- gated RMSNorm
// y = (w + w_offset) * x * rstd(x) * silu(g): the output norm of gated linear-attention blocks
// (Qwen3.5 GatedDeltaNet). One block per row; x is kept in registers between the two passes.
__global__ void __launch_bounds__(NORM_T)
    rmsnorm_gated_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ g,
                             const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                             float* __restrict__ rstd_out, int H, float eps, float w_offset) {
  __shared__ float sh[32];
  const long long row = blockIdx.x;
  float ss = 0.f;
  for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8) {
    float f[8];
    load8(x + row * H + i, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum<NORM_T>(ss, sh);
  const float rstd = rsqrtf(ss / H + eps);
  if (threadIdx.x == 0) rstd_out[row] = rstd;
  for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8) {
    float f[8], gv[8], wv[8];
    load8(x + row * H + i, f);
    load8(g + row * H + i, gv);
    load8(w + i, wv);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      f[j] = f[j] * rstd * (wv[j] + w_offset) * (gv[j] * sigmoid_fast(gv[j]));
    store8(y + row * H + i, f);
  }
}
// With n = x*rstd*(w+off) and s = silu(g):  dg = dy*n*silu'(g);  dn = dy*s;
// dx = rstd * (dn*(w+off) - xhat * mean(dn*(w+off)*xhat));  dw += dn * xhat.
__global__ void __launch_bounds__(NORM_T)
    rmsnorm_gated_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                             const __nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ w,
                             const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                             __nv_bfloat16* __restrict__ dg, float* __restrict__ dw, int H, int rows,
                             float w_offset) {
  __shared__ float sh[32];
  float dw_acc[4][8];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[a][j] = 0.f;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float dot = 0.f;
    for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8) {
      float a[8], b[8], c[8], gv[8];
      load8(dy + row * H + i, a);
      load8(x + row * H + i, b);
      load8(w + i, c);
      load8(g + row * H + i, gv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float s = gv[j] * sigmoid_fast(gv[j]);
        dot += a[j] * s * (c[j] + w_offset) * b[j] * rstd;
      }
    }
    dot = block_sum<NORM_T>(dot, sh) / H;
    int k = 0;
    for (int i = threadIdx.x * 8; i < H; i += NORM_T * 8, ++k) {
      float a[8], b[8], c[8], gv[8], ox[8], og[8];
      load8(dy + row * H + i, a);
      load8(x + row * H + i, b);
      load8(w + i, c);
      load8(g + row * H + i, gv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float sg = sigmoid_fast(gv[j]);
        const float s = gv[j] * sg;
        const float xhat = b[j] * rstd;
        const float wj = c[j] + w_offset;
        const float dn = a[j] * s;
        ox[j] = rstd * (dn * wj - xhat * dot);
        og[j] = a[j] * xhat * wj * sg * (1.f + gv[j] * (1.f - sg));
        if (dw) {
          if (k < 4) dw_acc[k][j] += dn * xhat;
          else atomicAdd(dw + i + j, dn * xhat);
        }
      }
      store8(dx + row * H + i, ox);
      store8(dg + row * H + i, og);
    }
  }
  if (dw) {
    int k = 0;
    for (int i = threadIdx.x * 8; i < H && k < 4; i += NORM_T * 8, ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dw + i + j, dw_acc[k][j]);
  }
}

// ---------------------------------------------------------------------------------- entropy
// One block per row of a [R, V] bf16 logits chunk: a single online pass keeps the running maximum
// m, Z = sum exp(z - m) and S = sum (z - m) exp(z - m); entropy = log Z - S / Z. lse is returned
// as well. (The RL trainers log the policy entropy per token without a [R, V] fp32 softmax.)
__global__ void __launch_bounds__(ENT_T)
    entropy_kernel(const __nv_bfloat16* __restrict__ logits, float* __restrict__ ent,
                   float* __restrict__ lse_out, int V, long long ld, float inv_temp) {
  __shared__ float sh[32];
  const long long r = blockIdx.x;
  const __nv_bfloat16* z = logits + r * ld;
  const int v8 = V & ~7;
  float m = -INFINITY, Z = 0.f, S = 0.f;
  auto push = [&](float v) {
    v *= inv_temp;
    if (v > m) {  // rescale the running sums to the new maximum
      const float c = __expf(m - v);
      S = (m == -INFINITY) ? 0.f : c * (S + (m - v) * Z);
      Z = (m == -INFINITY) ? 0.f : c * Z;
      m = v;
    }
    const float e = __expf(v - m);
    Z += e;
    S += (v - m) * e;
  };
  for (int i = threadIdx.x * 8; i < v8; i += ENT_T * 8) {
    float f[8];
    load8(z + i, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) push(f[j]);
  }
  for (int i = v8 + threadIdx.x; i < V; i += ENT_T) push(__bfloat162float(z[i]));
  const float M = block_max<ENT_T>(m, sh);
  const float c = (m == -INFINITY) ? 0.f : __expf(m - M);
  const float Zs = c * Z, Ss = c * (S + (m - M) * Z);
  const float Zt = block_sum<ENT_T>(Zs, sh);
  const float St = block_sum<ENT_T>((m == -INFINITY) ? 0.f : Ss, sh);
  if (threadIdx.x == 0) {
    ent[r] = logf(Zt) - St / Zt;
    if (lse_out) lse_out[r] = M + logf(Zt);  // of the scaled logits
  }
}

// ---------------------------------------------------------------------------------- optimizer
// Flat fp32 buffers, 16-byte accesses where every pointer allows them (`nv` vectors), single elements behind.
AXB_DEVICE bool axb_aligned16(const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; }

// sum of squares of a flat fp32 gradient buffer -> out[0] (atomic). Bound: HBM. Four vectors in
// flight: 307M elements 324 -> 199 us (6.2 TB/s).
__global__ void __launch_bounds__(256) sumsq_kernel(const float* __restrict__ g, long long n, float* __restrict__ out) {
  __shared__ float sh[32];
  const long long step = (long long)gridDim.x * 256, i0 = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long nv = axb_aligned16(g) ? n >> 2 : 0;
  float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long long i = i0; i < nv; i += 4 * step) {
    float4 a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      a[k] = i + k * step < nv ? reinterpret_cast<const float4*>(g)[i + k * step] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s4.x += a[k].x * a[k].x;
      s4.y += a[k].y * a[k].y;
      s4.z += a[k].z * a[k].z;
      s4.w += a[k].w * a[k].w;
    }
  }
  float s = (s4.x + s4.y) + (s4.z + s4.w);
  for (long long i = (nv << 2) + i0; i < n; i += step) s += g[i] * g[i];
  s = block_sum<256>(s, sh);
  if (threadIdx.x == 0) atomicAdd(out, s);
}
// y += s[0] * x, flat fp32. Bound: HBM (65.5M elements 120 us, 6.6 TB/s).
__global__ void __launch_bounds__(256) axpy_f32_kernel(float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ s,
                                                       long long n) {
  const float a = *s;
  const long long step = (long long)gridDim.x * 256, i0 = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long nv = axb_aligned16(x) && axb_aligned16(y) ? n >> 2 : 0;
  for (long long i = i0; i < nv; i += 2 * step) {
    float4 u[2], w[2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (i + k * step < nv) u[k] = reinterpret_cast<const float4*>(x)[i + k * step], w[k] = reinterpret_cast<float4*>(y)[i + k * step];
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (i + k * step < nv)
        reinterpret_cast<float4*>(y)[i + k * step] = make_float4(fmaf(a, u[k].x, w[k].x), fmaf(a, u[k].y, w[k].y),
                                                                 fmaf(a, u[k].z, w[k].z), fmaf(a, u[k].w, w[k].w));
  }
  for (long long i = (nv << 2) + i0; i < n; i += step) y[i] = fmaf(a, x[i], y[i]);
}
// Fused AdamW over a flat fp32 master buffer. gnorm_sq (device scalar, optional) drives clipping:
// grads are scaled by min(1, max_norm / (sqrt(gnorm_sq) + 1e-6)) without a host round trip.
// bf16_copy (optional) receives the updated parameters for the bf16 compute path.
// Bound: HBM, 30 bytes per parameter. One vector per thread and as many blocks as that takes: a bounded grid that strides is
// slower, whatever is in flight (150M parameters: 666 us = 6.8 TB/s; 148 x 16 blocks 735, two vectors in flight 750; 788 with
// single elements before).
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p, const float* __restrict__ g,
                             float* __restrict__ m, float* __restrict__ v,
                             __nv_bfloat16* __restrict__ bf16_copy, long long n, float lr,
                             float beta1, float beta2, float eps, float wd, float bc1, float bc2,
                             const float* __restrict__ gnorm_sq, float max_norm,
                             float grad_scale) {
  float clip = grad_scale;
  if (gnorm_sq && max_norm > 0.f) {
    const float nrm = sqrtf(*gnorm_sq) * grad_scale;
    clip *= fminf(1.f, max_norm / (nrm + 1e-6f));
  }
  auto update = [&](float& pi, float gi, float& mi, float& vi) {
    gi *= clip;
    mi = beta1 * mi + (1.f - beta1) * gi;
    vi = beta2 * vi + (1.f - beta2) * gi * gi;
    pi *= (1.f - lr * wd);
    pi -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  };
  const long long step = (long long)gridDim.x * 256, i0 = (long long)blockIdx.x * 256 + threadIdx.x;
  const bool al = axb_aligned16(p) && axb_aligned16(g) && axb_aligned16(m) && axb_aligned16(v) &&
                  (reinterpret_cast<uintptr_t>(bf16_copy) & 7) == 0;
  const long long nv = al ? n >> 2 : 0;
  for (long long i = i0; i < nv; i += step) {
    const float4 g4 = reinterpret_cast<const float4*>(g)[i];
    float4 p4 = reinterpret_cast<float4*>(p)[i], m4 = reinterpret_cast<float4*>(m)[i], v4 = reinterpret_cast<float4*>(v)[i];
    update(p4.x, g4.x, m4.x, v4.x);
    update(p4.y, g4.y, m4.y, v4.y);
    update(p4.z, g4.z, m4.z, v4.z);
    update(p4.w, g4.w, m4.w, v4.w);
    reinterpret_cast<float4*>(m)[i] = m4;
    reinterpret_cast<float4*>(v)[i] = v4;
    reinterpret_cast<float4*>(p)[i] = p4;
    if (bf16_copy) reinterpret_cast<uint2*>(bf16_copy)[i] = make_uint2(pack_bf16x2(p4.x, p4.y), pack_bf16x2(p4.z, p4.w));
  }
  for (long long i = (nv << 2) + i0; i < n; i += step) {
    float pi = p[i], mi = m[i], vi = v[i];
    update(pi, g[i], mi, vi);
    m[i] = mi;
    v[i] = vi;
    p[i] = pi;
    if (bf16_copy) bf16_copy[i] = __float2bfloat16(pi);
  }
}

// dst(bf16/fp32) = alpha * src (+ dst if accumulate)
__global__ void cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ s, float* __restrict__ d,
                                        long long n, float alpha, int accumulate) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float x = alpha * __bfloat162float(s[i]);
    d[i] = accumulate ? d[i] + x : x;
  }
}
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ s, __nv_bfloat16* __restrict__ d,
                                        long long n, float alpha) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    d[i] = __float2bfloat16(alpha * s[i]);
}
// y[i] += x[i]  (bf16, 8-wide)
__global__ void add_bf16_kernel(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x,
                                long long n8) {
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n8;
       v += (long long)gridDim.x * blockDim.x) {
    float a[8], b[8];
    load8(y + v * 8, a);
    load8(x + v * 8, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += b[j];
    store8(y + v * 8, a);
  }
}

inline int grid_for(long long work, int threads, int cap = 148 * 16) {
  long long g = (work + threads - 1) / threads;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}
}  // namespace

#define ST(s) reinterpret_cast<cudaStream_t>(s)

static int rmsnorm_fwd_launch(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd,
                              long long rows, int H, float eps, float w_offset, bool pdl, void* stream) {
  if (H % 8) return -2;
  if (rows <= 0) return 0;
  AxbLaunch l(dim3((unsigned)rows), NORM_T, 0, ST(stream), 0, pdl);
  const int nv = (H / 8 + NORM_T - 1) / NORM_T;
  auto kern = nv == 1 ? rmsnorm_fwd_kernel<1> : (nv == 2 ? rmsnorm_fwd_kernel<2> : (nv <= 4 ? rmsnorm_fwd_kernel<4> : rmsnorm_fwd_kernel<0>));
  const cudaError_t e = cudaLaunchKernelEx(&l.cfg, kern, (const __nv_bfloat16*)x, (const __nv_bfloat16*)res,
                                           (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (__nv_bfloat16*)res_out, rstd, H, eps,
                                           w_offset);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
extern "C" int axb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y,
                               void* res_out, float* rstd, long long rows, int H, float eps,
                               float w_offset, void* stream) {
  return rmsnorm_fwd_launch(x, res, w, y, res_out, rstd, rows, H, eps, w_offset, false, stream);
}
// the same as a dependent launch: it may start before its predecessor on the stream has finished, and waits for it
extern "C" int axb_rmsnorm_fwd_pdl(const void* x, const void* res, const void* w, void* y, void* res_out, long long rows,
                                   int H, float eps, float w_offset, void* stream) {
  return rmsnorm_fwd_launch(x, res, w, y, res_out, nullptr, rows, H, eps, w_offset, true, stream);
}
extern "C" int axb_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd,
                               const void* dres, void* dx, float* dw, long long rows, int H,
                               float w_offset, void* stream) {
  if (H % 8) return -2;
  if (rows <= 0) return 0;
  const int nv = (H / 8 + NORM_T - 1) / NORM_T;
  auto kern = rmsnorm_bwd_wide_kernel;
  int per_sm = 8;
  if (nv <= 4) {
    kern = nv == 1 ? (dw ? rmsnorm_bwd_kernel<1, true> : rmsnorm_bwd_kernel<1, false>)
         : nv == 2 ? (dw ? rmsnorm_bwd_kernel<2, true> : rmsnorm_bwd_kernel<2, false>)
                   : (dw ? rmsnorm_bwd_kernel<4, true> : rmsnorm_bwd_kernel<4, false>);
    per_sm = nv == 4 ? 2 : 4;      // resident blocks: their row loops keep the loads in flight, more only add flushes
  }
  const int grid = rows < 148 * per_sm ? (int)rows : 148 * per_sm;
  kern<<<grid, NORM_T, 0, ST(stream)>>>(
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)h, (const __nv_bfloat16*)w, rstd,
      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, dw, H, (int)rows, w_offset);
  return (int)cudaGetLastError();
}
extern "C" int axb_rope_qk(void* qkv, const int* pos, const float* inv_freq, int T, int Hq, int Hk,
                           int D, long long row_stride, float sign, float attn_scale,
                           const void* qn_w, const void* kn_w, float* rstd_out, float eps,
                           void* stream) {
  if (T <= 0) return 0;
  if (!qn_w && !kn_w && (D % 4) == 0 && (row_stride % 2) == 0) {
    rope_fast_kernel<<<rope_grid(T, Hq + Hk), 256, 0, ST(stream)>>>((__nv_bfloat16*)qkv, pos, inv_freq, T, Hq + Hk, D,
                                                                     row_stride, sign, attn_scale, D);
    return (int)cudaGetLastError();
  }
  const long long warps = (long long)T * (Hq + Hk);
  const int wpb = 8;
  rope_qk_kernel<<<(unsigned)((warps + wpb - 1) / wpb), wpb * 32, 0, ST(stream)>>>(
      (__nv_bfloat16*)qkv, pos, inv_freq, T, Hq, Hk, D, row_stride, sign, attn_scale,
      (const __nv_bfloat16*)qn_w, (const __nv_bfloat16*)kn_w, rstd_out, eps);
  return (int)cudaGetLastError();
}
// Partial rotary embedding of the first `rot` dimensions of the q and k heads (sign = -1: the inverse rotation,
// i.e. the backward pass). rot % 4 == 0, rot <= D, row_stride % 2 == 0.
extern "C" int axb_rope_partial(void* qkv, const int* pos, const float* inv_freq, int T, int n_heads, int D, int rot,
                                long long row_stride, float sign, float attn_scale, void* stream) {
  if (T <= 0) return 0;
  if (rot <= 0 || rot > D || (rot & 3) || (row_stride & 1) || (D & 1)) return -2;
  rope_fast_kernel<<<rope_grid(T, n_heads), 256, 0, ST(stream)>>>((__nv_bfloat16*)qkv, pos, inv_freq, T, n_heads, D,
                                                                   row_stride, sign, attn_scale, rot);
  return (int)cudaGetLastError();
}
extern "C" int axb_rope_qk_bwd(void* dqkv, const void* x_pre, const int* pos,
                               const float* inv_freq, int T, int Hq, int Hk, int D,
                               long long row_stride, long long x_row_stride, float attn_scale,
                               const void* qn_w, const void* kn_w, const float* rstd_in,
                               float* dqn_w, float* dkn_w, void* stream) {
  if (T <= 0) return 0;
  if (D > 512) return -2;
  if (!qn_w && !kn_w && (D % 4) == 0 && (row_stride % 2) == 0) {
    rope_fast_kernel<<<rope_grid(T, Hq + Hk), 256, 0, ST(stream)>>>((__nv_bfloat16*)dqkv, pos, inv_freq, T, Hq + Hk, D,
                                                                     row_stride, -1.f, attn_scale, D);
    return (int)cudaGetLastError();
  }
  const long long warps = (long long)T * (Hq + Hk);
  const int wpb = 8;
  if (D <= 256)
    rope_qk_bwd_kernel<4><<<(unsigned)((warps + wpb - 1) / wpb), wpb * 32, 0, ST(stream)>>>(
        (__nv_bfloat16*)dqkv, (const __nv_bfloat16*)x_pre, pos, inv_freq, T, Hq, Hk, D, row_stride,
        x_row_stride, attn_scale, (const __nv_bfloat16*)qn_w, (const __nv_bfloat16*)kn_w, rstd_in,
        dqn_w, dkn_w);
  else      // Gemma 4's global layers: 512-wide heads
    rope_qk_bwd_kernel<8><<<(unsigned)((warps + wpb - 1) / wpb), wpb * 32, 0, ST(stream)>>>(
        (__nv_bfloat16*)dqkv, (const __nv_bfloat16*)x_pre, pos, inv_freq, T, Hq, Hk, D, row_stride,
        x_row_stride, attn_scale, (const __nv_bfloat16*)qn_w, (const __nv_bfloat16*)kn_w, rstd_in,
        dqn_w, dkn_w);
  return (int)cudaGetLastError();
}
extern "C" int axb_rmsnorm_gated_fwd(const void* x, const void* g, const void* w, void* y,
                                     float* rstd, long long rows, int H, float eps,
                                     float w_offset, void* stream) {
  if (H % 8) return -2;
  if (rows <= 0) return 0;
  rmsnorm_gated_fwd_kernel<<<(unsigned)rows, NORM_T, 0, ST(stream)>>>(
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)g, (const __nv_bfloat16*)w,
      (__nv_bfloat16*)y, rstd, H, eps, w_offset);
  return (int)cudaGetLastError();
}
extern "C" int axb_rmsnorm_gated_bwd(const void* dy, const void* x, const void* g, const void* w,
                                     const float* rstd, void* dx, void* dg, float* dw,
                                     long long rows, int H, float w_offset, void* stream) {
  if (H % 8) return -2;
  if (rows <= 0) return 0;
  const unsigned grid = (unsigned)(rows < 148 * 4 ? rows : 148 * 4);
  rmsnorm_gated_bwd_kernel<<<grid, NORM_T, 0, ST(stream)>>>(
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)g,
      (const __nv_bfloat16*)w, rstd, (__nv_bfloat16*)dx, (__nv_bfloat16*)dg, dw, H, (int)rows,
      w_offset);
  return (int)cudaGetLastError();
}
extern "C" int axb_entropy(const void* logits, float* ent, float* lse, long long rows, int V,
                           long long ld, float inv_temp, void* stream) {
  if (rows <= 0) return 0;
  if (ld % 8) return -2;
  entropy_kernel<<<(unsigned)rows, ENT_T, 0, ST(stream)>>>((const __nv_bfloat16*)logits, ent, lse, V,
                                                         ld, inv_temp);
  return (int)cudaGetLastError();
}
extern "C" int axb_dora_norm(const float* WA, const float* B, const float* G, const float* w2, float* norm, long long N,
                             int R, float s, void* stream) {
  if (N <= 0) return 0;
  if (R < 1 || R > 128) return -2;
  dora_norm_kernel<<<(unsigned)((N + 127) / 128), 128, R * R * sizeof(float), ST(stream)>>>(WA, B, G, w2, norm, N, R, s);
  return (int)cudaGetLastError();
}

extern "C" int axb_glu_fwd(const void* gu, void* h, long long T, int I, int kind, float limit,
                           void* stream) {
  if (I % 8) return -2;
  if (T <= 0) return 0;
  glu_fwd_kernel<<<grid_for(T * (I / 8), 256), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)gu, (__nv_bfloat16*)h, T, I, kind, limit, nullptr);
  return (int)cudaGetLastError();
}
// the same over the first *blocks_in_use * 128 rows only (device-side count)
extern "C" int axb_glu_fwd_rows(const void* gu, void* h, long long T, int I, int kind, float limit,
                                const int* blocks_in_use, void* stream) {
  if (I % 8) return -2;
  if (T <= 0) return 0;
  glu_fwd_kernel<<<grid_for(T * (I / 8), 256), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)gu, (__nv_bfloat16*)h, T, I, kind, limit, blocks_in_use);
  return (int)cudaGetLastError();
}
extern "C" int axb_glu_bwd_rows(const void* dh, const void* gu, void* dgu, long long T, int I, int kind,
                                float limit, const int* blocks_in_use, void* stream) {
  if (I % 8) return -2;
  if (T <= 0) return 0;
  glu_bwd_kernel<<<grid_for(T * (I / 8), 256), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)dh, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, T, I, kind, limit, blocks_in_use);
  return (int)cudaGetLastError();
}
extern "C" int axb_glu_bwd(const void* dh, const void* gu, void* dgu, long long T, int I, int kind,
                           float limit, void* stream) {
  if (I % 8) return -2;
  if (T <= 0) return 0;
  glu_bwd_kernel<<<grid_for(T * (I / 8), 256), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)dh, (const __nv_bfloat16*)gu, (__nv_bfloat16*)dgu, T, I, kind, limit, nullptr);
  return (int)cudaGetLastError();
}
extern "C" int axb_embedding_fwd(const void* table, const long long* ids, void* out, long long T,
                                 int H, long long vocab, void* stream) {
  if (H % 8) return -2;
  if (T <= 0) return 0;
  embedding_fwd_kernel<<<grid_for(T * (H / 8), 256), 256, 0, ST(stream)>>>(
      (const __nv_bfloat16*)table, ids, (__nv_bfloat16*)out, T, H, vocab);
  return (int)cudaGetLastError();
}
extern "C" int axb_embedding_bwd(const void* dout, const long long* ids, float* dtable,
                                 long long T, int H, long long vocab, void* stream) {
  if (T <= 0) return 0;
  const __nv_bfloat16* d = (const __nv_bfloat16*)dout;
  if (H % 8 == 0 && ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dtable)) & 15) == 0)
    embedding_bwd_kernel<8><<<grid_for(T * (H / 8), 256), 256, 0, ST(stream)>>>(d, ids, dtable, T, H, vocab);
  else
    embedding_bwd_kernel<1><<<grid_for(T * H, 256), 256, 0, ST(stream)>>>(d, ids, dtable, T, H, vocab);
  return (int)cudaGetLastError();
}
extern "C" int axb_ce_fwd_bwd(void* logits, const long long* labels, float* loss, float* lse,
                              long long rows, int V, long long ld, float grad_scale,
                              long long ignore_index, int write_grad, void* stream) {
  if (rows <= 0) return 0;
  if (ld % 8) return -2;
  return ce_launch<false>(logits, labels, loss, lse, rows, V, ld, grad_scale, ignore_index, write_grad, 0.f, ST(stream));
}
// the same with soft-capped logits, z' = softcap * tanh(z / softcap)
extern "C" int axb_ce_fwd_bwd_softcap(void* logits, const long long* labels, float* loss, float* lse,
                                      long long rows, int V, long long ld, float grad_scale,
                                      long long ignore_index, int write_grad, float softcap, void* stream) {
  if (rows <= 0) return 0;
  if (ld % 8 || !(softcap > 0.f)) return -2;
  return ce_launch<true>(logits, labels, loss, lse, rows, V, ld, grad_scale, ignore_index, write_grad, softcap, ST(stream));
}
extern "C" int axb_axpy_f32(float* y, const float* x, const float* s, long long n, void* stream) {
  if (n <= 0) return 0;
  axpy_f32_kernel<<<grid_for(n / 4 + 1, 256), 256, 0, ST(stream)>>>(y, x, s, n);
  return (int)cudaGetLastError();
}
extern "C" int axb_sumsq(const float* g, long long n, float* out, void* stream) {
  if (n <= 0) return 0;
  sumsq_kernel<<<grid_for(n / 4 + 1, 256, 148 * 6), 256, 0, ST(stream)>>>(g, n, out);
  return (int)cudaGetLastError();
}
extern "C" int axb_adamw(float* p, const float* g, float* m, float* v, void* bf16_copy,
                         long long n, float lr, float beta1, float beta2, float eps, float wd,
                         float bc1, float bc2, const float* gnorm_sq, float max_norm,
                         float grad_scale, void* stream) {
  if (n <= 0) return 0;
  adamw_kernel<<<grid_for(n / 4 + 1, 256, 1 << 30), 256, 0, ST(stream)>>>(p, g, m, v, (__nv_bfloat16*)bf16_copy, n,
                                                         lr, beta1, beta2, eps, wd, bc1, bc2,
                                                         gnorm_sq, max_norm, grad_scale);
  return (int)cudaGetLastError();
}
extern "C" int axb_cast_bf16_to_f32(const void* s, float* d, long long n, float alpha,
                                    int accumulate, void* stream) {
  if (n <= 0) return 0;
  cast_bf16_to_f32_kernel<<<grid_for(n, 256), 256, 0, ST(stream)>>>((const __nv_bfloat16*)s, d, n,
                                                                    alpha, accumulate);
  return (int)cudaGetLastError();
}
extern "C" int axb_cast_f32_to_bf16(const float* s, void* d, long long n, float alpha,
                                    void* stream) {
  if (n <= 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n, 256), 256, 0, ST(stream)>>>(s, (__nv_bfloat16*)d, n,
                                                                    alpha);
  return (int)cudaGetLastError();
}
extern "C" int axb_add_bf16(void* y, const void* x, long long n, void* stream) {
  if (n % 8) return -2;
  if (n <= 0) return 0;
  add_bf16_kernel<<<grid_for(n / 8, 256), 256, 0, ST(stream)>>>((__nv_bfloat16*)y,
                                                                (const __nv_bfloat16*)x, n / 8);
  return (int)cudaGetLastError();
}
