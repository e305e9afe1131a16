"""Generation steps, one host call per decoder layer (csrc/decode_step.cu).

A step of a few token rows is bound by the weights it reads, tens of microseconds a layer, and the operator-by-operator
path costs the interpreter several times that. Layers whose every part is the plain form of the architecture (RMS norms,
rotary attention with optional per-head norms, gated MLP, optional LoRA) are launched as a whole; every other layer, and
every model with hooks or wrappers on a part, keeps its own ``forward``.
"""
from __future__ import annotations

import ctypes as C

import torch
from torch.nn.modules import module as _nn

from ..ops import _lib
from ..ops.functional import _ACT_KIND
from .layers import FusedLinear, RMSNorm, adapters_enabled

_vp, _i32, _i64, _f32 = C.c_void_p, C.c_int, C.c_longlong, C.c_float


class _Proj(C.Structure):
    _fields_ = [("W", _vp), ("bias", _vp), ("A", _vp), ("B", _vp), ("N", _i32), ("K", _i32), ("rank", _i32), ("scaling", _f32)]


class _Layer(C.Structure):
    _fields_ = ([(n, _Proj) for n in ("qkv", "o", "gate_up", "down")]
                + [(n, _vp) for n in ("norm1", "norm2", "q_norm", "k_norm", "x", "res_in", "res_mid", "res_out", "y", "xn", "qkv_buf",
                                      "att", "gu", "act", "low", "k_cache", "v_cache", "seq", "lens", "pos", "inv_freq")]
                + [(n, _i64) for n in ("max_len", "rows")]
                + [(n, _i32) for n in ("B", "Hq", "Hk", "D", "window", "glu_kind", "chained", "pad")]
                + [(n, _f32) for n in ("eps1", "off1", "eps2", "off2", "attn_scale", "scale", "norm_eps", "glu_limit")]
                + [("status", _vp)])


_lib.register_cuda_sigs({"axb_decode_layer": [_vp, _vp]})

MAX_ROWS = 128      # beyond, the 128-row tiles of the ordinary GEMM are full and its path is the faster one


# Everything below runs once per layer and step, next to launches that take a few microseconds each: submodules and
# parameters are read from the modules' own dictionaries, which costs a tenth of nn.Module's attribute lookup.
def _bare(m, cls):
    return type(m) is cls and "forward" not in m.__dict__ and not m._forward_hooks and not m._forward_pre_hooks


def _dense16(t):
    return t.dtype == torch.bfloat16 and t.is_cuda and t.is_contiguous() and t.data_ptr() % 16 == 0


def _proj(p, m, adapters):
    """Fills ``p`` from a projection; False where it is not a dense one with at most a plain LoRA adapter."""
    d = m.__dict__
    if not _bare(m, FusedLinear) or m.dora_magnitude is not None or m.mora_M is not None or d["qat"] is not None:
        return False
    w, bias, A = m._parameters["weight"], m.bias, m.lora_A
    extra = w.__dict__
    if "_axb_quant" in extra or "_axb_shard" in extra or w.dim() != 2 or not _dense16(w):
        return False
    N, K = w.shape
    if N % 8 or K % 8 or (bias is not None and not _dense16(bias)):
        return False
    p.W, p.bias, p.N, p.K, p.rank = w.data_ptr(), None if bias is None else bias.data_ptr(), N, K, 0
    if A is not None and not d["merged"] and adapters:
        if d["lora_dropout"] > 0.0 and d["training"]:
            return False
        if m.lora_A16 is None:
            m.refresh_shadows()
        A16, B16 = m.lora_A16, m.lora_B16
        if not _dense16(A16) or not _dense16(B16) or A16.shape[0] % 8 or B16.shape != (N, A16.shape[0]):
            return False
        p.A, p.B, p.rank, p.scaling = A16.data_ptr(), B16.data_ptr(), A16.shape[0], float(d["scaling"])
    return True


def _norm_ok(m, dim):
    w = m._parameters["weight"] if _bare(m, RMSNorm) else None
    return w is not None and w.numel() == dim and _dense16(w)


def _plain_layer(layer):
    """(attention, MLP) of a decoder layer in the plain form, or None."""
    from .transformer import MLP, Attention, DecoderLayer

    if not _bare(layer, DecoderLayer):
        return None
    d, sub = layer.__dict__, layer._modules
    if (d["is_moe"] or d["parallel_block"] or d["post_norm_only"] or d["sandwich"] or d["residual_multiplier"] != 1.0
            or layer.layer_scalar is not None or d["ple_width"] or layer.g4_moe is not None):
        return None
    a, f = sub["self_attn"], sub["mlp"]
    if not _bare(a, Attention) or not _bare(f, MLP):
        return None
    e, g = a.__dict__, f.__dict__
    if (e["k_eq_v"] or e["kv_store"] or e["kv_src"] is not None or a.sinks is not None or a.out_gate is not None or e["clip_qkv"]
            or e["norm_after_rope"] or e["full_qk_norm"] or e["v_norm"] or not e["use_rope"] or e["rot_dim"] is not None
            or e["softcap"] or e["llama4"] or e["chunk"] or e["temp"] is not None or e["q_pos_scale"] is not None
            or g["gate_multiplier"] != 1.0 or g["down_multiplier"] != 1.0):
        return None
    if e["D"] not in (64, 128, 256) or e["Hq"] % e["Hk"] or e["Hq"] // e["Hk"] > 16:
        return None
    return a, f


class DecodeStep:
    """The layers of one generation step. ``layer(...)`` returns (branch output, residual stream, None), or None for a
    layer that has to run its own ``forward``. The returned tensors are this step's own buffers: the next layer's call
    overwrites them."""

    @staticmethod
    def of(model, h, pos, meta):
        """A step for this pass, or None where nothing of it can run this way."""
        from .kv_cache import KVCache

        cache = getattr(meta, "kv_cache", None)
        if (cache is None or not getattr(meta, "decode", False) or not h.is_cuda or h.dtype != torch.bfloat16 or model.hooks is not None
                or torch.is_grad_enabled() or h.dim() != 2 or not 0 < h.shape[0] <= MAX_ROWS):
            return None
        if type(cache) is not KVCache or "attend" in cache.__dict__ or not (_dense16(cache.k) and _dense16(cache.v)):
            return None
        if _nn._global_forward_hooks or _nn._global_forward_pre_hooks:
            return None
        for t, dtype in ((meta.seq, torch.int64), (meta.lens_after, torch.int32), (pos, torch.int32)):     # one per row, as the kernels read them
            if not torch.is_tensor(t) or t.dtype != dtype or t.device != h.device or t.shape != h.shape[:1]:
                return None
        return DecodeStep(h, pos, meta)

    def __init__(self, h, pos, meta):
        self.B, self.H = h.shape
        c = self.cache = meta.kv_cache
        self.keep = [pos.contiguous(), meta.seq.contiguous(), meta.lens_after.contiguous()]
        self.bytes = {}
        self.y, self.res = torch.empty_like(h), torch.empty_like(h)
        self.last = None            # the branch output this step produced last: the next launch may overlap its producer
        self.lib = _lib.cuda_lib()
        self.stream = _lib.stream_ptr()
        self.k_ptr, self.v_ptr, self.layer_bytes = c.k.data_ptr(), c.v.data_ptr(), c.k.stride(0) * 2
        s = self.s = _Layer()
        s.pos, s.seq, s.lens = (t.data_ptr() for t in self.keep)
        s.B, s.rows, s.max_len, s.status = self.B, c.k.shape[1], c.k.shape[2], _lib.status_word(h.device).data_ptr()
        s.y, s.res_out = self.y.data_ptr(), self.res.data_ptr()
        self.adapters = adapters_enabled()
        self.sized = None

    def _size(self, shape, h):
        """Scratch rows for layers of these widths (kept for the step: nearly always one set for all layers)."""
        W, O, I, gu, rank = shape
        cols = (self.H, self.H, W, O, I, gu, rank)
        at = [0]
        for c in cols:
            at.append(at[-1] + (self.B * c + 63) // 64 * 64)
        t = torch.empty(at[-1], dtype=torch.bfloat16, device=h.device)
        self.keep.append(t)
        s, base = self.s, t.data_ptr()
        s.res_mid, s.xn, s.qkv_buf, s.att, s.act, s.gu, s.low = (base + 2 * a for a in at[:-1])
        self.sized = shape

    def layer(self, layer, h, residual, inv_freq, attn_scale):
        parts = _plain_layer(layer)
        if parts is None or not h.is_contiguous() or (residual is not None and not residual.is_contiguous()):
            return None
        a, f = parts
        e, sub, s = a.__dict__, layer._modules, self.s
        Hq, Hk, D, on = e["Hq"], e["Hk"], e["D"], self.adapters
        gate_up = f._modules["gate_up_proj"]
        if not (_proj(s.qkv, a._modules["qkv_proj"], on) and _proj(s.o, a._modules["o_proj"], on) and _proj(s.gate_up, gate_up, on)
                and _proj(s.down, f._modules["down_proj"], on)):
            return None
        n1, n2 = sub["input_layernorm"], sub["post_attention_layernorm"]
        qn, kn = a.q_norm, a.k_norm
        if not _norm_ok(n1, self.H) or not _norm_ok(n2, self.H) or (qn is None) != (kn is None):
            return None
        if qn is not None and (not _norm_ok(qn, D) or not _norm_ok(kn, D) or qn.offset or kn.offset):
            return None
        if a.local_inv_freq is not None:
            inv_freq, attn_scale = a.local_inv_freq, 1.0
        I, W = s.gate_up.N // 2, (Hq + 2 * Hk) * D
        if (s.qkv.K != self.H or s.qkv.N != W or s.o.K != Hq * D or s.o.N != self.H or s.gate_up.K != self.H or s.down.K != I
                or s.down.N != self.H or self.cache.width != Hk * D or e["layer_idx"] >= self.cache.L
                or inv_freq.dtype != torch.float32 or not inv_freq.is_contiguous()):
            return None
        kind = _ACT_KIND[f.act]
        fused = I % 64 == 0 and kind < 2 and gate_up.bias is None
        shape = (W, Hq * D, I, 0 if fused else 2 * I, max(s.qkv.rank, s.o.rank, s.gate_up.rank, s.down.rank))
        if shape != self.sized:
            self._size(shape, h)
        s.norm1, s.norm2 = n1._parameters["weight"].data_ptr(), n2._parameters["weight"].data_ptr()
        s.q_norm, s.k_norm = (None, None) if qn is None else (qn._parameters["weight"].data_ptr(), kn._parameters["weight"].data_ptr())
        s.x, s.res_in = h.data_ptr(), _lib.ptr(residual)
        at = e["layer_idx"] * self.layer_bytes
        s.k_cache, s.v_cache, s.inv_freq = self.k_ptr + at, self.v_ptr + at, inv_freq.data_ptr()
        s.Hq, s.Hk, s.D, s.window = Hq, Hk, D, int(e["window"] or 0)
        s.glu_kind, s.glu_limit = kind, float(f.glu_limit or 0.0)
        s.chained = int(self.last is not None and self.last is h)
        s.eps1, s.off1, s.eps2, s.off2 = n1.eps, n1.offset, n2.eps, n2.offset
        s.attn_scale, s.scale, s.norm_eps = attn_scale, e["scale"], e["eps"]
        _lib.check_rc(self.lib.axb_decode_layer(C.addressof(s), self.stream), "decode_layer")
        self.last = self.y
        return self.y, self.res, None
