"""Kernels of a generation step against plain PyTorch: decode attention over the KV cache."""
import math

import pytest
import torch

from axolotl_b200.ops import functional as Fn

pytestmark = pytest.mark.gpu


def _rotate(x, pos, inv_freq):
    a = pos.float()[:, None, None] * inv_freq
    c, s = a.cos(), a.sin()
    h = x.shape[-1] // 2
    x1, x2 = x[..., :h].float(), x[..., h:].float()
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).to(x.dtype)


def _reference(q, k, v, scale, first, n):
    """fp32 attention of [Hk, G, D] queries over rows first..n of [rows, Hk, D] caches."""
    kk, vv = (t[first:n].float().transpose(0, 1) for t in (k, v))
    return (torch.softmax(q.float() @ kk.transpose(1, 2) * scale, -1) @ vv).reshape(-1)


@pytest.mark.parametrize("D,Hq,Hk", [(64, 8, 8), (64, 32, 4), (128, 32, 8), (128, 32, 2), (256, 8, 2), (128, 15, 3)])
@pytest.mark.parametrize("splits", [0, 1, 2, 8])
@pytest.mark.parametrize("window", [0, 33])
@pytest.mark.parametrize("append,rope", [(False, False), (True, False), (True, True)])
def test_decode_attention_splits_append_and_rope(D, Hq, Hk, splits, window, append, rope):
    """Lengths at the edges of a warp's 16-position tile and of a cluster's stride; cache rows in another order than the
    queries; rows past the end hold NaN, which must not reach the result. Bound: the output is one bf16 rounding of an
    fp32 result (2^-8 of its largest element covers it with the rotated operands' own rounding)."""
    from axolotl_b200.ops import _lib

    torch.manual_seed(D + Hq + splits)
    lens = [1, 2, 15, 16, 17, 64, 65, 500, 511]
    B, cap = len(lens), 520
    W = (Hq + 2 * Hk) * D
    qkv = torch.randn(B, W + 8, device="cuda").bfloat16()[:, :W]       # a row stride of its own
    kc, vc = (torch.randn(B, cap, Hk * D, device="cuda").bfloat16() for _ in range(2))
    seq = torch.randperm(B, device="cuda")
    n = torch.tensor(lens, dtype=torch.int32, device="cuda")
    for b in range(B):
        kc[seq[b], lens[b]:], vc[seq[b], lens[b]:] = float("nan"), float("nan")
        if append:
            kc[seq[b], lens[b] - 1], vc[seq[b], lens[b] - 1] = float("nan"), float("nan")
    pos = (n - 1).contiguous()
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    scale = 1.0 / math.sqrt(D)
    out = torch.full((B, Hq * D), 7.0, device="cuda", dtype=torch.bfloat16)
    k0, v0 = kc.clone(), vc.clone()
    _lib.check_rc(_lib.cuda_lib().axb_decode_attn(
        qkv.data_ptr(), qkv.stride(0), 0, Hq * D, (Hq + Hk) * D, kc.data_ptr(), vc.data_ptr(), seq.data_ptr(), n.data_ptr(),
        pos.data_ptr(), inv.data_ptr() if rope else None, 1.0, out.data_ptr(), out.stride(0), B, Hq, Hk, D, cap, scale, window,
        int(append), splits, 0, _lib.stream_ptr()), "decode_attn")
    q = qkv[:, :Hq * D].reshape(B, Hq, D)
    k = qkv[:, Hq * D:(Hq + Hk) * D].reshape(B, Hk, D)
    v = qkv[:, (Hq + Hk) * D:].reshape(B, Hk, D)
    if rope:
        q, k = _rotate(q, pos, inv), _rotate(k, pos, inv)
    for b in range(B):
        if append:
            k0[seq[b], lens[b] - 1], v0[seq[b], lens[b] - 1] = k[b].reshape(-1), v[b].reshape(-1)
        ref = _reference(q[b].view(Hk, Hq // Hk, D), k0[seq[b]].view(cap, Hk, D), v0[seq[b]].view(cap, Hk, D), scale,
                         max(0, lens[b] - window) if window else 0, lens[b])
        assert torch.isfinite(out[b].float()).all()
        assert (out[b].float() - ref).abs().max() <= 2 ** -8 * max(1.0, ref.abs().max().item()), lens[b]
    if append:      # the new rows are in the cache (a rotated value may round the other way), every other row is untouched
        torch.testing.assert_close(vc, v0, rtol=0, atol=0, equal_nan=True)
        torch.testing.assert_close(kc, k0, rtol=2 ** -7, atol=2 ** -7 if rope else 0, equal_nan=True)


@pytest.mark.parametrize("cap,n", [(256, 200), (120, 100)])
def test_decode_attention_with_scores_of_minus_infinity(cap, n):
    """A whole 16-position tile (first, middle or last) whose scores are -inf has weight 0, with one CTA per pair and with four."""
    torch.manual_seed(n)
    B, Hq, Hk, D = 3, 8, 2, 64
    qkv = torch.randn(B, (Hq + 2 * Hk) * D, device="cuda").bfloat16()
    qkv[:, 0:Hq * D:D] = 1.0
    k, v = torch.randn(2, B, cap, Hk * D, device="cuda").bfloat16()
    for b, p0 in enumerate((0, 48, n - n % 16)):
        k[b, p0:p0 + 16, 0::D] = float("-inf")
    lens = torch.full((B,), n, dtype=torch.int32, device="cuda")
    scale = D ** -0.5
    out = Fn.decode_attention(qkv, k, v, lens, Hq, Hk, D, scale)
    for b in range(B):
        q = qkv[b, :Hq * D].view(Hk, Hq // Hk, D).float()
        kk, vv = (t[b, :n].view(n, Hk, D).float().transpose(0, 1) for t in (k, v))
        s = (q @ kk.transpose(1, 2) * scale)
        ref = (torch.softmax(s, -1) @ vv).reshape(-1)
        assert torch.isfinite(ref).all()
        assert (out[b].float() - ref).abs().max() <= 2 ** -8 * max(1.0, ref.abs().max().item())


def test_cached_step_on_a_subset_of_the_sequences():
    """``KVCache.attend`` with query rows that belong to some of the cache's sequences, in another order."""
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import KVCache, _DecodeMeta
    from axolotl_b200.models.transformer import CausalLM

    m = CausalLM(preset("tiny-llama", num_hidden_layers=1), dtype=torch.bfloat16, device="cuda").init_weights(0)
    a = m.layers[0].self_attn
    cache = KVCache(m, 5, 40)
    cache.k.normal_()
    cache.v.normal_()
    k0, v0 = cache.k[0].clone(), cache.v[0].clone()
    seq = torch.tensor([3, 0, 4], device="cuda")
    pos = torch.tensor([7, 0, 39], device="cuda")
    qkv = torch.randn(3, (a.Hq + 2 * a.Hk) * a.D, device="cuda").bfloat16()
    out = cache.attend(0, qkv, _DecodeMeta(cache, seq, pos, False), a.Hq, a.Hk, a.D, a.scale)
    nq, nk = a.Hq * a.D, a.Hk * a.D
    k0[seq, pos], v0[seq, pos] = qkv[:, nq:nq + nk], qkv[:, nq + nk:]
    assert torch.equal(cache.k[0], k0) and torch.equal(cache.v[0], v0)
    ref = Fn.decode_attention(qkv.cpu(), k0[seq].cpu(), v0[seq].cpu(), (pos + 1).int().cpu(), a.Hq, a.Hk, a.D, a.scale)
    assert (out.cpu().float() - ref.float()).abs().max() <= 2 ** -7 * max(1.0, ref.abs().max().item())


_SEQ_FORMS = {
    "int32": lambda t: t.int(),
    "strided": lambda t: torch.stack([t, t.flip(0)], 1)[:, 0],
    "host": lambda t: t.cpu(),
    "list": lambda t: t.tolist(),
}


@pytest.mark.parametrize("form", sorted(_SEQ_FORMS))
@pytest.mark.parametrize("whole_model", [False, True])
def test_cached_step_takes_the_sequence_ids_of_an_indexed_store(form, whole_model):
    """Sequence ids of another integer type, stride or device than the kernel's own: the same result and the same cache, bit for bit."""
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import KVCache, _DecodeMeta
    from axolotl_b200.models.transformer import CausalLM

    torch.manual_seed(1)
    m = CausalLM(preset("tiny-llama", vocab_size=512, num_hidden_layers=1), dtype=torch.bfloat16, device="cuda").init_weights(0).eval()
    a = m.layers[0].self_attn
    ids = torch.tensor([3, 0, 4, 1], device="cuda")
    pos = torch.tensor([7, 0, 39, 12], device="cuda")
    qkv = torch.randn(4, (a.Hq + 2 * a.Hk) * a.D, device="cuda").bfloat16()
    kv = torch.randn(2, 1, 5, 40, a.Hk * a.D, device="cuda").bfloat16()
    got = []
    for seq in (ids, _SEQ_FORMS[form](ids)):
        cache = KVCache(m, 5, 40)
        cache.k.copy_(kv[0])
        cache.v.copy_(kv[1])
        meta = _DecodeMeta(cache, seq, pos, False)
        with torch.no_grad():
            if whole_model:    # a step of another form than the one-call layers take runs operator by operator: a rounding apart
                out = m(torch.arange(4, device="cuda")[None], pos.int()[None], attn_meta=meta, return_logits=False).hidden_states
            else:
                out = cache.attend(0, qkv, meta, a.Hq, a.Hk, a.D, a.scale)
        got.append((out, cache.k, cache.v))
    for x, y in zip(*got):
        assert torch.equal(x, y) if not whole_model else ((x.float() - y.float()).norm() <= 0.012 * y.float().norm())


@pytest.mark.parametrize("bad", [torch.zeros(4), torch.zeros(3, dtype=torch.long), torch.zeros(4, 1, dtype=torch.long)])
def test_cached_step_refuses_other_sequence_ids(bad):
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import KVCache, _DecodeMeta
    from axolotl_b200.models.transformer import CausalLM

    m = CausalLM(preset("tiny-llama", num_hidden_layers=1), dtype=torch.bfloat16, device="cuda")
    a, cache = m.layers[0].self_attn, KVCache(m, 5, 40)
    qkv = torch.zeros(4, (a.Hq + 2 * a.Hk) * a.D, device="cuda").bfloat16()
    with pytest.raises(IndexError):
        cache.attend(0, qkv, _DecodeMeta(cache, bad.cuda(), torch.arange(4, device="cuda"), False), a.Hq, a.Hk, a.D, a.scale)


def _in_checked_library(test):
    """Runs a test of this file again with the bounds-check library."""
    import os
    import subprocess
    import sys

    if os.environ.get("AXB_BOUNDS_CHECK") != "1":
        r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "no:cacheprovider", f"{__file__}::{test}"],
                           env=dict(os.environ, AXB_BOUNDS_CHECK="1"), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stdout[-3000:]


def test_cached_step_outside_the_cache_stores_nothing():
    """Positions and rows at and past the cache's ends: only the rows inside are stored (negative ones count from the end, as
    an indexed store has it), the others give zeros, their neighbours stay as they are, and the status word tells."""
    from axolotl_b200.ops import _lib

    torch.manual_seed(2)
    B, cap, Hq, Hk, D = 4, 20, 8, 2, 64
    big = torch.randn(2, B + 4, cap, Hk * D, device="cuda").bfloat16()      # cache rows 0..3 with two rows around them
    k, v = big[0, 2:2 + B], big[1, 2:2 + B]
    seq = torch.tensor([0, 3, -1, 4, -5, 1, 2, 2], device="cuda")
    pos = torch.tensor([cap, 19, 5, 3, 3, 2 ** 30, -1, -cap - 1], device="cuda")
    good = {1: (3, 19), 2: (3, 5), 6: (2, 19)}
    qkv = torch.randn(8, (Hq + 2 * Hk) * D, device="cuda").bfloat16()
    want = big.clone()
    for i, (r, p) in good.items():
        want[0, 2 + r, p], want[1, 2 + r, p] = qkv[i, Hq * D:(Hq + Hk) * D], qkv[i, (Hq + Hk) * D:]
    out = Fn.decode_attention_append(qkv, k, v, seq, (pos + 1).int(), Hq, Hk, D, D ** -0.5)
    if _lib.cuda_lib().axb_bounds_check_enabled():
        v0 = _lib.bounds_violation()
        assert v0 is not None and v0[0] in ("KV cache row", "KV cache position") and v0[3] == 5, v0
    with pytest.raises(_lib.KernelBoundsError):
        _lib.check_status()
    _lib.check_status()
    assert torch.equal(big, want)
    for i in range(8):
        if i not in (1, 2):
            assert not out[i].any()
    i = 2
    ref = _reference(qkv[i, :Hq * D].view(Hk, Hq // Hk, D), want[0, 5].view(cap, Hk, D), want[1, 5].view(cap, Hk, D), D ** -0.5, 0, 6)
    assert (out[i].float() - ref).abs().max() <= 2 ** -8 * max(1.0, ref.abs().max().item())
    assert out[1].any()
    _in_checked_library("test_cached_step_outside_the_cache_stores_nothing")


@pytest.mark.parametrize("R,N,K,K2", [(128, 1, 64, 0), (200, 5, 72, 16), (1000, 17, 520, 48), (6144, 64, 4096, 0), (129, 100, 640, 8),
                                      (384, 256, 1032, 64)])
@pytest.mark.parametrize("splits", [0, 1, 3, 8])
@pytest.mark.parametrize("mode,f32", [(0, False), (0, True), (1, False), (1, True), (2, False)])
def test_skinny_gemm(R, N, K, K2, splits, mode, f32):
    """Remainders of the 128-row tile, of the 64-wide K block and of the short side, all cluster sizes. fp32 sums in another
    order: 2^-20 of the accumulated magnitude; bf16 results one rounding more (2^-8)."""
    from axolotl_b200.ops import _lib

    torch.manual_seed(R + N)
    if mode == 2:
        R = (R + 63) // 64 * 64
    rows = 2 * R if mode == 2 else R
    P, S = torch.randn(rows, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    P2 = torch.randn(rows, K2, device="cuda").bfloat16() if K2 else None
    S2 = torch.randn(N, K2, device="cuda").bfloat16() if K2 else None
    bias = torch.randn(R, device="cuda").bfloat16() if mode == 0 else None
    acc = S.double() @ P.double().t()
    mag = S.double().abs() @ P.double().abs().t()
    if K2:
        acc, mag = acc + S2.double() @ P2.double().t(), mag + S2.double().abs() @ P2.double().abs().t()
    acc, mag = acc * 0.5, mag * 0.5
    if bias is not None:
        acc = acc + bias.double()
    if mode == 2:
        g, u = acc.chunk(2, -1)
        ref = torch.nn.functional.silu(g) * u
        tol = 2 ** -8 * ref.abs() + 2 ** -8 * (1 + g.abs() + u.abs()) * 2 ** -6 + 2 ** -14 * mag.chunk(2, -1)[0]
    else:
        ref, tol = acc, 2 ** -20 * mag + (0 if f32 else 2 ** -8 * acc.abs())
    if mode == 1:
        ref, tol = ref.t(), tol.t()
    ld = ref.shape[1] + 3                                  # an odd output stride
    buf = torch.full((ref.shape[0], ld), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    _lib.check_rc(_lib.cuda_lib().axb_gemm_skinny(
        P.data_ptr(), K, S.data_ptr(), K, buf.data_ptr(), ld, R, N, K, _lib.ptr(P2), K2, _lib.ptr(S2), K2, K2, 0.5,
        _lib.ptr(bias), mode, int(f32), 0, 0.0, 1, splits, 0, _lib.status_word().data_ptr(), _lib.stream_ptr()), "gemm_skinny")
    _lib.check_status()
    out = buf[:, :ref.shape[1]].double()
    assert ((out - ref).abs() <= tol + 1e-30).all(), ((out - ref).abs() - tol).max()
    assert (buf[:, ref.shape[1]:] == 7.0).all()


@pytest.mark.parametrize("M,N,K,skinny", [(129, 31, 512, True), (20000, 16, 512, True), (300, 32, 768, True), (300, 32, 760, False),
                                          (4224, 64, 1536, True), (4232, 64, 1536, False), (4232, 64, 5120, True), (11784, 64, 5120, False),
                                          (16, 512, 512, True), (32, 4232, 2048, True), (32, 11784, 1024, False), (64, 4224, 1280, True),
                                          (64, 4232, 1280, False), (128, 4232, 5120, True), (128, 4232, 5112, False)])
def test_short_side_products_on_both_sides_of_the_rule(M, N, K, skinny):
    """Sizes just inside and outside the lines between the short-side kernel and the ordinary tiles. fp32 sums in any order:
    2^-20 of their magnitude, one bf16 rounding more for the result."""
    from axolotl_b200.ops import _lib
    from axolotl_b200.ops.gemm import _use_skinny, gemm

    torch.manual_seed(M)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    out = gemm(a, b)
    assert _use_skinny(M, N, K, False, False, out, 0, None, 0.0) == skinny
    _lib.check_status()
    ref, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    assert ((out.double() - ref).abs() <= 2 ** -20 * mag + 2 ** -8 * ref.abs()).all()


_STEP_CASES = {
    "llama": dict(),
    "qwen3 q/k norms": dict(model_type="qwen3", head_dim=64),
    "qwen2 biases": dict(model_type="qwen2", attention_bias=True),
    "gelu, odd width": dict(hidden_act="gelu_pytorch_tanh", intermediate_size=360),
    "window": dict(model_type="mistral", extra=dict(sliding_window=24)),
    "wide groups": dict(num_attention_heads=8, num_key_value_heads=1, head_dim=128),
}


@pytest.mark.parametrize("name", sorted(_STEP_CASES))
@pytest.mark.parametrize("batch,lora", [(1, False), (8, True), (33, False), (128, True)])
def test_decode_layers_in_one_call_match_the_operator_path(name, batch, lora, monkeypatch):
    """Hidden states, logits and cache of a step against the layer-by-layer operators; both round every intermediate to bf16,
    so the difference is a few roundings (2^-8 each) of a normalised stream through three layers."""
    from axolotl_b200.models import decode_step
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import KVCache, _DecodeMeta
    from axolotl_b200.models.lora import ALL_LINEAR, LoraSpec, inject_lora
    from axolotl_b200.models.transformer import CausalLM

    torch.manual_seed(3)
    cfg = preset("tiny-llama", vocab_size=512, num_hidden_layers=3, **_STEP_CASES[name])
    m = CausalLM(cfg, dtype=torch.bfloat16, device="cuda").init_weights(0)
    if lora:
        inject_lora(m, LoraSpec(r=8, lora_alpha=16, target_modules=[t for t in ALL_LINEAR if t != "k_proj"]))
    with torch.no_grad():
        for n, p in m.named_parameters():
            if "lora_B" in n or n.endswith("bias"):
                p.normal_(0, 0.05)
        for f in m.modules():
            if getattr(f, "lora_B", None) is not None:     # off-diagonal blocks stay zero
                keep = torch.zeros_like(f.lora_B)
                for r0, rows, c0, cols in f.lora_blocks:
                    keep[r0:r0 + rows, c0:c0 + cols] = 1
                f.lora_B.mul_(keep)
    m.refresh_lora_shadows()
    m.eval()
    lens = torch.randint(0, 60, (batch,))
    pos = lens.cuda()
    seq = torch.randperm(batch, device="cuda")
    tok = torch.randint(0, 512, (batch,), device="cuda")
    outs = []
    k, v = torch.randn(2, 3, batch, 64, m.layers[0].self_attn.Hk * m.layers[0].self_attn.D, device="cuda").bfloat16()
    for fused in (True, False):
        cache = KVCache(m, batch, 64)
        cache.k.copy_(k)
        cache.v.copy_(v)
        calls = []
        if not fused:
            monkeypatch.setattr(decode_step.DecodeStep, "of", staticmethod(lambda *a: None))
        else:
            real = decode_step.DecodeStep.layer
            monkeypatch.setattr(decode_step.DecodeStep, "layer", lambda self, *a: calls.append(real(self, *a)) or calls[-1])
        with torch.no_grad():
            o = m(tok[None], pos.int()[None], attn_meta=_DecodeMeta(cache, seq, pos, False), return_logits=True, capture_hidden=[1, 2])
        outs.append((o.logits.float(), o.hidden_states.float(), o.captured[2].float(), cache.k.float(), cache.v.float()))
        if fused:
            assert len(calls) == 3 and all(c is not None for c in calls)
            monkeypatch.undo()
    for a, b in zip(*outs):
        assert ((a - b).norm() / b.norm()).item() < 0.012 and torch.isfinite(a).all()


# (config, adapter, layers that have to run their own forward)
_OWN_FORWARD = {
    "experts beside dense layers": (dict(model_type="qwen3_moe", num_experts=8, num_experts_per_tok=2, moe_intermediate_size=128,
                                         mlp_only_layers=[0, 2]), None, {1}),
    "adapters disabled": (dict(), dict(), set()),
    "adapters merged": (dict(), dict(), set()),
    "magnitude-decomposed adapters": (dict(), dict(use_dora=True), {0, 1, 2}),
    "square adapters": (dict(), dict(use_mora=True), {0, 1, 2}),
    "4-bit weight": (dict(), None, {1}),
    "partial rotation": (dict(extra=dict(partial_rotary_factor=0.5)), None, {0, 1, 2}),
    "norms on the branch outputs too": (dict(model_type="glm4"), None, {0, 1, 2}),
    "norms on the branch outputs only": (dict(model_type="olmo2", qk_norm=True), None, {0, 1, 2}),
    "attention and MLP side by side": (dict(model_type="cohere"), None, {0, 1, 2}),
    "scaled branches": (dict(model_type="granite", extra=dict(residual_multiplier=0.5)), None, {0, 1, 2}),
    "a layer without rotation": (dict(model_type="smollm3", extra=dict(no_rope_layers=[1, 0, 1])), None, {1}),
    "adapter dropout while training": (dict(), dict(lora_dropout=0.3), {0, 1, 2}),
}


@pytest.mark.parametrize("name", sorted(_OWN_FORWARD))
def test_decode_step_leaves_other_layers_to_their_own_forward(name, monkeypatch):
    """Layers that are not of the plain form: which of them refuse the one-call form, and the step's result against a step whose
    layers all run their own forward (a few bf16 roundings apart where some do not)."""
    from axolotl_b200.models import decode_step
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import KVCache, _DecodeMeta
    from axolotl_b200.models.layers import FusedLinear, disable_adapters
    from axolotl_b200.models.lora import ALL_LINEAR, LoraSpec, inject_lora
    from axolotl_b200.models.transformer import CausalLM

    over, adapter, own = _OWN_FORWARD[name]
    torch.manual_seed(5)
    m = CausalLM(preset("tiny-llama", vocab_size=512, num_hidden_layers=3, **over), dtype=torch.bfloat16, device="cuda").init_weights(0).eval()
    if adapter is not None:
        inject_lora(m, LoraSpec(r=8, lora_alpha=16, target_modules=list(ALL_LINEAR), **adapter))
        with torch.no_grad():
            for n, p in m.named_parameters():
                if "lora_B" in n or "mora_M" in n:
                    p.normal_(0, 0.05)
            for f in m.modules():
                if getattr(f, "lora_B", None) is not None:
                    keep = torch.zeros_like(f.lora_B)
                    for r0, rows, c0, cols in f.lora_blocks:
                        keep[r0:r0 + rows, c0:c0 + cols] = 1
                    f.lora_B.mul_(keep)
        m.refresh_lora_shadows()
    if name == "adapters merged":
        for f in m.modules():
            if isinstance(f, FusedLinear):
                f.merge_lora_()
    if name == "4-bit weight":
        m.layers[1].mlp.down_proj.quantize_nf4_()
    training = name == "adapter dropout while training"
    m.train(training)
    pos = torch.randint(0, 60, (8,), device="cuda")
    tok = torch.randint(0, 512, (8,), device="cuda")
    at = m.layers[0].self_attn
    k, v = torch.randn(2, 3, 8, 64, at.Hk * at.D, device="cuda").bfloat16()
    done, outs = [], []
    real = decode_step.DecodeStep.layer
    monkeypatch.setattr(decode_step.DecodeStep, "layer", lambda self, *a: done.append(real(self, *a) if not force else None) or done[-1])
    for force in (False, True):
        cache = KVCache(m, 8, 64)
        cache.k.copy_(k)
        cache.v.copy_(v)
        meta = _DecodeMeta(cache, torch.arange(8, device="cuda"), pos, True)
        with torch.no_grad():
            if name == "adapters disabled":
                with disable_adapters():
                    o = m(tok[None], pos.int()[None], attn_meta=meta, return_logits=True)
            else:
                o = m(tok[None], pos.int()[None], attn_meta=meta, return_logits=True)
        outs.append((o.logits.float(), cache.k.float(), cache.v.float()))
    assert {i for i in range(3) if done[i] is None} == own and len(done) == 6
    for a, b in zip(*outs):
        assert torch.isfinite(a).all()
        if not training:
            assert torch.equal(a, b) if len(own) == 3 else ((a - b).norm() <= 0.012 * b.norm())


def test_decode_step_leaves_a_hooked_layer_to_its_own_forward():
    """A forward hook inside a layer is called on every pass."""
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import generate_cached
    from axolotl_b200.models.transformer import CausalLM

    m = CausalLM(preset("tiny-llama", vocab_size=512), dtype=torch.bfloat16, device="cuda").init_weights(0)
    a = generate_cached(m, [[1, 5, 9], [7, 8]], 6)
    seen = []
    h = m.layers[1].mlp.down_proj.register_forward_hook(lambda mod, i, o: seen.append(o.shape[0]))
    b = generate_cached(m, [[1, 5, 9], [7, 8]], 6)
    h.remove()
    assert len(seen) == 6 and a == b


@pytest.mark.parametrize("M,N", [(129, 256), (129, 4096), (256, 320), (257, 2056), (300, 1000), (511, 4096), (640, 14336)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("c_in", [False, True])
def test_gemm_tiles_chosen_below_512_rows(M, N, ta, tb, c_in):
    """Problems that the CTA-pair kernel used to refuse: few rows, few tiles, ragged edges, all operand layouts and the
    accumulating epilogue. fp32 sums of 264 products: 2^-20 of their magnitude."""
    from axolotl_b200.ops import _lib
    from axolotl_b200.ops.gemm import _pick_tile, gemm

    torch.manual_seed(M + N)
    K = 264
    if (ta and M % 8) or (tb and N % 8):
        pytest.skip("a transposed operand needs 16-byte rows")
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    aa, bb = a.t().contiguous() if ta else a, b.t().contiguous() if tb else b
    ref, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    c = torch.randn(M, N, device="cuda") if c_in else None
    want = ref + c.double() if c_in else ref
    out = gemm(aa, bb, trans_a=ta, trans_b=tb, out_dtype=torch.float32, c_in=c, beta=1.0 if c_in else 0.0)
    assert ((out.double() - want).abs() <= 2 ** -20 * (mag + want.abs())).all(), _pick_tile(M, N)
    if not c_in:
        o16 = gemm(aa, bb, trans_a=ta, trans_b=tb)
        assert ((o16.double() - ref).abs() <= 2 ** -20 * mag + 2 ** -8 * ref.abs()).all()
    _lib.check_status()


@pytest.mark.parametrize("M,N,K,out,tile", [(1568, 2712, 88, 0, (256, True)), (1304, 3720, 96, 2, (64, False)), (200, 300, 136, 1, (64, False)),
                                            (3824, 264, 920, 2, (128, False)), (300, 37000, 72, 1, (256, False)), (1032, 1056, 392, 0, (256, True))])
def test_gemm_tiles_by_waves_and_epilogue(M, N, K, out, tile):
    """Every tile width by its own rule, with the epilogue that decides for it (bf16, fp32, added to fp32). fp32 sums: 2^-20 of
    their magnitude, one bf16 rounding more for bf16."""
    from axolotl_b200.ops import _lib
    from axolotl_b200.ops.gemm import _pick_tile, gemm

    assert _pick_tile(M, N, (K + 63) // 64, out) == tile
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    ref, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    if out == 2:
        c = torch.randn(M, N, device="cuda")
        ref, mag = ref + c.double(), mag + c.double().abs()
        got = gemm(a, b, out=c, accumulate=True)
    else:
        got = gemm(a, b, out_dtype=torch.float32 if out else torch.bfloat16)
    _lib.check_status()
    assert ((got.double() - ref).abs() <= 2 ** -20 * mag + (0 if out else 2 ** -8 * ref.abs())).all()


@pytest.mark.parametrize("M,N,K", [(8, 512, 256), (16, 4096, 8192), (48, 1000, 960), (64, 14336, 328), (40, 777 * 8, 1000)])
@pytest.mark.parametrize("splits", [1, 3])
def test_gemm_accumulates_the_transposed_tile(M, N, K, splits):
    """t^T x into a strided fp32 buffer with a short first side. Atomic fp32 sums in any order: 2^-20 of their magnitude."""
    from axolotl_b200.ops import _lib
    from axolotl_b200.ops.gemm import gemm

    torch.manual_seed(M + N)
    t, x = torch.randn(K, M, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    buf = torch.randn(M, N + 4, device="cuda")
    c0 = buf.clone()
    gemm(t, x, trans_a=True, trans_b=True, out=buf[:, :N], accumulate=True, splits=splits, alpha=0.5)
    _lib.check_status()
    ref = c0[:, :N].double() + 0.5 * (t.double().t() @ x.double())
    mag = c0[:, :N].double().abs() + 0.5 * (t.double().abs().t() @ x.double().abs())
    assert ((buf[:, :N].double() - ref).abs() <= 2 ** -20 * mag).all() and torch.equal(buf[:, N:], c0[:, N:])


@pytest.mark.parametrize("width", [8, 256, 264, 1024])
def test_prompt_rows_go_to_their_cache_slots(width):
    from axolotl_b200.ops import _lib

    T, B, cap = 37, 5, 20
    qkv = torch.randn(T, 3 * width + 8, device="cuda").bfloat16()
    slots = torch.randperm(B * cap, device="cuda")[:T]
    seq, pos = slots // cap, slots % cap
    kc, vc = torch.randn(2, B, cap, width, device="cuda").bfloat16()
    k0, v0 = kc.clone(), vc.clone()
    _lib.check_rc(_lib.cuda_lib().axb_kv_append(qkv.data_ptr(), qkv.stride(0), width, 2 * width, kc.data_ptr(), vc.data_ptr(), seq.data_ptr(),
                                                pos.data_ptr(), T, width, B, cap, _lib.stream_ptr()), "kv_append")
    k0[seq, pos], v0[seq, pos] = qkv[:, width:2 * width], qkv[:, 2 * width:3 * width]
    assert torch.equal(kc, k0) and torch.equal(vc, v0)


@pytest.mark.parametrize("form", ["int64", "int32", "host", "list"])
def test_prompt_rows_take_the_indexes_of_an_indexed_store(form):
    """Sequence ids and positions of any integer form, negative ones counted from the end; rows of an odd stride."""
    from axolotl_b200.models.config import preset
    from axolotl_b200.models.kv_cache import KVCache, _PrefillMeta
    from axolotl_b200.models.transformer import CausalLM

    m = CausalLM(preset("tiny-llama", num_hidden_layers=1), dtype=torch.bfloat16, device="cuda")
    a, cache = m.layers[0].self_attn, KVCache(m, 5, 40)
    T, nq, nk = 24, a.Hq * a.D, a.Hk * a.D
    qkv = torch.randn(T, nq + 2 * nk, device="cuda").bfloat16()
    slots = torch.randperm(200, device="cuda")[:T]
    seq, pos = slots // 40 - 5 * (slots % 2), slots % 40 - 40 * (slots % 3 == 0)
    k0, v0 = cache.k.clone(), cache.v.clone()
    k0[0, seq, pos], v0[0, seq, pos] = qkv[:, nq:nq + nk], qkv[:, nq + nk:]
    f = {"int64": lambda t: t, "int32": lambda t: t.int(), "host": lambda t: t.cpu(), "list": lambda t: t.tolist()}[form]
    cache.attend(0, qkv, _PrefillMeta(cache, Fn.AttnMeta([0, T], "cuda"), f(seq), f(pos)), a.Hq, a.Hk, a.D, a.scale)
    assert torch.equal(cache.k, k0) and torch.equal(cache.v, v0)


def test_prompt_rows_outside_the_cache_are_not_stored():
    from axolotl_b200.ops import _lib

    T, B, cap, width = 6, 4, 20, 64
    qkv = torch.randn(T, 3 * width, device="cuda").bfloat16()
    big = torch.randn(2, B + 4, cap, width, device="cuda").bfloat16()
    k, v = big[0, 2:2 + B], big[1, 2:2 + B]
    seq = torch.tensor([0, B, -B - 1, 1, 2, 3], device="cuda")
    pos = torch.tensor([cap, 3, 3, -cap - 1, 2 ** 40, 7], device="cuda")
    want = big.clone()
    want[0, 5, 7], want[1, 5, 7] = qkv[5, width:2 * width], qkv[5, 2 * width:]
    _lib.check_rc(_lib.cuda_lib().axb_cache_append(
        qkv.data_ptr(), qkv.stride(0), width, 2 * width, k.data_ptr(), v.data_ptr(), seq.data_ptr(), pos.data_ptr(), T, width, B, cap,
        _lib.status_word().data_ptr(), _lib.stream_ptr()), "kv_append")
    if _lib.cuda_lib().axb_bounds_check_enabled():
        v0 = _lib.bounds_violation()
        assert v0 is not None and v0[0] in ("KV cache row", "KV cache position") and v0[3] == 5, v0
    with pytest.raises(_lib.KernelBoundsError):
        _lib.check_status()
    assert torch.equal(big, want)
    _in_checked_library("test_prompt_rows_outside_the_cache_are_not_stored")
