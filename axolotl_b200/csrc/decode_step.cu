// One decoder layer of a generation step (a few token rows against a KV cache) as one host call.
//
// A step at batch 8 streams a layer's weights in tens of microseconds, less than the interpreter needs to issue the layer's
// operators one by one, so the launches are issued from here: norm, qkv, attention (rotary embedding and cache append
// inside), o, norm, gate | up (gated activation inside), down, plus one small product per adapted projection. Every launch
// after the first is a dependent launch: its weight tiles are requested while its predecessor drains.
#include "axb_common.cuh"

extern "C" int axb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd, long long rows,
                               int H, float eps, float w_offset, void* stream);
extern "C" int axb_rmsnorm_fwd_pdl(const void* x, const void* res, const void* w, void* y, void* res_out, long long rows, int H,
                                   float eps, float w_offset, void* stream);
extern "C" int axb_gemm_skinny(const void* P, long long ldp, const void* S, long long lds, void* C, long long ldc, int R, int N,
                               int K, const void* P2, long long ldp2, const void* S2, long long lds2, int K2, float alpha,
                               const void* bias, int out_mode, int out_f32, int glu_kind, float glu_limit, int p_dep, int splits,
                               int pdl, int* status, void* stream);
extern "C" int axb_cache_attend(const void* qkv, long long ld, int q_col0, int k_col0, int v_col0, void* k_cache, void* v_cache,
                                long long rows, const long long* seq, const int* lens, const int* pos, const float* inv_freq,
                                float attn_scale, void* out, long long out_ld, int B, int Hq, int Hk, int D, long long max_len,
                                float scale, int window, int append, int splits, int pdl, int* status, void* stream);
extern "C" int axb_rope_qk(void* qkv, const int* pos, const float* inv_freq, int T, int Hq, int Hk, int D, long long row_stride,
                           float sign, float attn_scale, const void* qn_w, const void* kn_w, float* rstd_out, float eps,
                           void* stream);
extern "C" int axb_glu_fwd(const void* gu, void* h, long long T, int I, int kind, float limit, void* stream);

// A projection y = x W^T (+ bias) (+ s (x A^T) B^T); A [rank, K], B [N, rank] row-major bf16, rank 0: no adapter.
struct AxbDecodeProj {
  const void* W;
  const void* bias;
  const void* A;
  const void* B;
  int N, K, rank;
  float scaling;
};

// Filled by models/decode_step.py field by field, in this order.
struct AxbDecodeLayer {
  AxbDecodeProj qkv, o, gate_up, down;
  const void* norm1;
  const void* norm2;
  const void* q_norm;      // per-head norms (null: none)
  const void* k_norm;
  const void* x;           // branch output of the layer below, [B, H]
  const void* res_in;      // residual stream, null in the first layer (the stream is x itself)
  void* res_mid;           // stream after the first norm's addition (unused when res_in is null)
  void* res_out;           // stream after the second
  void* y;                 // [B, H]: branch output
  void* xn;                // scratch [B, H]
  void* qkv_buf;           // scratch [B, (Hq + 2 Hk) D]
  void* att;               // scratch [B, Hq D]
  void* gu;                // scratch [B, 2 I] (only where the activation is not fused)
  void* act;               // scratch [B, I]
  void* low;               // scratch [B, max rank]
  void* k_cache;
  void* v_cache;
  const long long* seq;
  const int* lens;
  const int* pos;
  const float* inv_freq;
  long long max_len, rows; // of the cache: positions per row, rows
  int B, Hq, Hk, D, window, glu_kind, chained, pad;
  float eps1, off1, eps2, off2, attn_scale, scale, norm_eps, glu_limit;
  int* status;
};

namespace {

// y = x W^T with an optional adapter; glu: y = act(gate) * up
int project(const AxbDecodeProj& p, const void* x, void* y, int B, void* low, bool glu, int kind, float limit, int* status,
            void* stream) {
  if (p.rank > 0) {
    const int rc = axb_gemm_skinny(p.A, p.K, x, p.K, low, p.rank, p.rank, B, p.K, nullptr, 0, nullptr, 0, 0, p.scaling, nullptr, 0,
                                   0, 0, 0.f, 0, 0, 1, status, stream);
    if (rc) return rc;
  }
  const int R = glu ? p.N / 2 : p.N;
  return axb_gemm_skinny(p.W, p.K, x, p.K, y, R, R, B, p.K, p.rank > 0 ? p.B : nullptr, p.rank, p.rank > 0 ? low : nullptr, p.rank,
                         p.rank, 1.f, p.bias, glu ? 2 : 0, 0, kind, limit, 0, 0, 1, status, stream);
}

}  // namespace

extern "C" int axb_decode_layer(const AxbDecodeLayer* l, void* stream) {
  const int B = l->B, H = l->qkv.K;
  int rc = l->chained ? axb_rmsnorm_fwd_pdl(l->x, l->res_in, l->norm1, l->xn, l->res_in ? l->res_mid : nullptr, B, H, l->eps1,
                                            l->off1, stream)
                      : axb_rmsnorm_fwd(l->x, l->res_in, l->norm1, l->xn, l->res_in ? l->res_mid : nullptr, nullptr, B, H,
                                        l->eps1, l->off1, stream);
  const void* mid = l->res_in ? l->res_mid : l->x;
  if (!rc) rc = project(l->qkv, l->xn, l->qkv_buf, B, l->low, false, 0, 0.f, l->status, stream);
  const int nq = l->Hq * l->D, nk = l->Hk * l->D, W = nq + 2 * nk;
  const bool qk_norm = l->q_norm != nullptr || l->k_norm != nullptr;
  if (!rc && qk_norm)
    rc = axb_rope_qk(l->qkv_buf, l->pos, l->inv_freq, B, l->Hq, l->Hk, l->D, W, 1.f, l->attn_scale, l->q_norm, l->k_norm, nullptr,
                     l->norm_eps, stream);
  if (!rc)
    rc = axb_cache_attend(l->qkv_buf, W, 0, nq, nq + nk, l->k_cache, l->v_cache, l->rows, l->seq, l->lens, l->pos,
                          qk_norm ? nullptr : l->inv_freq, l->attn_scale, l->att, nq, B, l->Hq, l->Hk, l->D, l->max_len, l->scale,
                          l->window, 1, 0, qk_norm ? 0 : 1, l->status, stream);
  if (!rc) rc = project(l->o, l->att, l->y, B, l->low, false, 0, 0.f, l->status, stream);
  if (!rc) rc = axb_rmsnorm_fwd_pdl(l->y, mid, l->norm2, l->xn, l->res_out, B, H, l->eps2, l->off2, stream);
  const int I = l->gate_up.N / 2;
  const bool fused = I % 64 == 0 && (l->glu_kind == 0 || l->glu_kind == 1) && !l->gate_up.bias;
  if (!rc) rc = project(l->gate_up, l->xn, fused ? l->act : l->gu, B, l->low, fused, l->glu_kind, l->glu_limit, l->status, stream);
  if (!rc && !fused) rc = axb_glu_fwd(l->gu, l->act, B, I, l->glu_kind, l->glu_limit, stream);
  if (!rc) rc = project(l->down, l->act, l->y, B, l->low, false, 0, 0.f, l->status, stream);
  return rc;
}
