"""RMSNorm and attention kernels at the edges of their per-thread vectors and block tiles, against PyTorch."""
import numpy as np
import pytest
import torch

from axolotl_b200.ops import _lib
from axolotl_b200.ops import functional as Fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 1000, 2048, 2056, 4096, 5120, 8192, 8200, 16392])
@pytest.mark.parametrize("rows", [1, 7, 593, 1300])
@pytest.mark.parametrize("res", [False, True])
@pytest.mark.parametrize("dw", [False, True])
def test_rmsnorm_kernels(H, rows, res, dw):
    """H at and beside one, two and four vectors per thread and beyond; rows below, at and above the resident blocks. y and
    dx are one bf16 rounding of an fp32 row result; dw sums `rows` fp32 terms in another order."""
    torch.manual_seed(H + rows)
    lib, st = _lib.cuda_lib(), _lib.stream_ptr()
    x, r, dy = (torch.randn(rows, H, device="cuda").bfloat16() for _ in range(3))
    w = torch.randn(H, device="cuda").bfloat16()
    y, h, dx = (torch.full((rows + 1, H), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    rstd = torch.empty(rows, device="cuda")
    _lib.check_rc(lib.axb_rmsnorm_fwd(x.data_ptr(), r.data_ptr() if res else None, w.data_ptr(), y.data_ptr(),
                                      h.data_ptr() if res else None, rstd.data_ptr(), rows, H, 1e-5, 0.5, st), "rmsnorm_fwd")
    hh = (x.float() + r.float()).bfloat16() if res else x
    if res:
        assert torch.equal(h[:rows], hh)
    hd = hh.double()
    rs = torch.rsqrt(hd.pow(2).mean(-1, keepdim=True) + 1e-5)
    wd = w.double() + 0.5
    ref = hd * rs * wd
    assert ((y[:rows].double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all() and (y[rows:] == 7).all()
    g = torch.randn(H, device="cuda") if dw else None
    g0 = g.double() if dw else None
    _lib.check_rc(lib.axb_rmsnorm_bwd(dy.data_ptr(), hh.data_ptr(), w.data_ptr(), rstd.data_ptr(), r.data_ptr() if res else None,
                                      dx.data_ptr(), _lib.ptr(g), rows, H, 0.5, st), "rmsnorm_bwd")
    xh, dyd = hd * rs, dy.double()
    gd = dyd * wd
    want = rs * (gd - xh * (gd * xh).mean(-1, keepdim=True)) + (r.double() if res else 0)
    big = rs * (gd.abs() + xh.abs() * (gd * xh).abs().mean(-1, keepdim=True)) + (r.double().abs() if res else 0)
    assert ((dx[:rows].double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -18 * big).all() and (dx[rows:] == 7).all()
    if dw:
        t = dyd * xh
        assert ((g.double() - g0 - t.sum(0)).abs() <= 2 ** -18 * (t.abs().sum(0) + g0.abs())).all()


@pytest.mark.parametrize("D,Hq,Hk", [(64, 3, 1), (64, 9, 9), (64, 16, 2), (128, 12, 2), (128, 5, 5)])
@pytest.mark.parametrize("lens", [[1], [31, 2], [33, 64, 130], [400, 257]])
@pytest.mark.parametrize("window,causal", [(0, True), (70, True), (0, False)])
def test_attention_head_and_token_remainders(D, Hq, Hk, lens, window, causal):
    """Head counts that are not multiples of a block's, odd and even groups, lengths around the 32-, 64-, 128- and 256-row
    tiles: output and gradients against fp32 autograd. bf16 operands, probabilities and gradients: 2^-6 of the largest
    element, 2^-7 in the norm."""
    torch.manual_seed(D + Hq)
    T = sum(lens)
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda").bfloat16().requires_grad_(True)
    do = torch.randn(T, Hq * D, device="cuda").bfloat16()
    meta = Fn.AttnMeta(np.concatenate([[0], np.cumsum(lens)]), "cuda", causal)
    meta = meta.windowed(window) if window else meta
    o = Fn.flash_varlen(qkv, meta, Hq, Hk, D)
    (g,) = torch.autograd.grad(o, qkv, do)
    x = qkv.detach().float().requires_grad_(True)
    q, k, v = (t.reshape(T, -1, D) for t in x.split([Hq * D, Hk * D, Hk * D], -1))
    ref = Fn._attn_ref(q, k, v, meta.cu_seqlens_host, D ** -0.5, causal, window).reshape(T, -1)
    (gr,) = torch.autograd.grad(ref, x, do.float())
    for a, b in ((o.detach().float(), ref.detach()), (g.float(), gr)):
        assert ((a - b).abs() <= 2 ** -6 * b.abs().max()).all()
        assert ((a - b).norm() / b.norm()).item() < 2 ** -7
    _lib.check_status()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lens", [[3], [4], [1, 130], [2, 131, 64], [3, 97, 35], [32, 32, 5, 129]])
def test_attention_gradient_of_queries_by_row_alignment(D, lens):
    """The sums of dQ leave in groups of four rows: documents that begin at every place of a group, buffers that end inside one, and the
    queries of a rank that begin inside a tile (its sums before that row are not its own). Rows of the query gradient against the fp32
    reference as in test_attention_head_and_token_remainders; nothing behind the scratch is written."""
    import axolotl_b200.parallel.cp  # noqa: F401  (declares the entry for a rank's rows)

    torch.manual_seed(D + sum(lens))
    Hq, Hk, T, lib, st = 4, 2, sum(lens), _lib.cuda_lib(), _lib.stream_ptr()
    qkv, do = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda").bfloat16(), torch.randn(T, Hq * D, device="cuda").bfloat16()
    cu = np.concatenate([[0], np.cumsum(lens)])
    meta = Fn.AttnMeta(cu, "cuda")
    x = qkv.float().requires_grad_(True)
    q, k, v = (t.reshape(T, -1, D) for t in x.split([Hq * D, Hk * D, Hk * D], -1))
    (want,) = torch.autograd.grad(Fn._attn_ref(q, k, v, meta.cu_seqlens_host, D ** -0.5, True, 0).reshape(T, -1), x, do.float())
    out, lse = torch.empty_like(do), torch.empty(Hq, T, device="cuda")
    word = _lib.status_word(qkv.device).data_ptr()
    _lib.check_rc(lib.axb_flash_varlen_fwd(qkv.data_ptr(), qkv.stride(0), T, Hq, Hk, D, 0, Hq * D, (Hq + Hk) * D, meta.tiles_fwd.data_ptr(),
                                           meta.n_tiles, out.data_ptr(), out.stride(0), lse.data_ptr(), D ** -0.5, word, st), "fwd")
    kv = qkv[:, Hq * D:].contiguous()
    for off, n in ((0, T), (T // 3, T - T // 3), (T // 2, 1)):
        acc = torch.full((n * Hq * D + 64,), 5.0, device="cuda")
        dqkv, delta = torch.zeros(T, qkv.shape[1], device="cuda", dtype=torch.bfloat16), torch.empty(Hq, n, device="cuda")
        rows = lambda t: t[off:off + n].contiguous()  # noqa: E731
        ql, dl, ol, ll = rows(qkv), rows(do), rows(out), lse[:, off:off + n].contiguous()
        if (off, n) == (0, T):
            rc = lib.axb_flash_varlen_bwd(ql.data_ptr(), ql.stride(0), dl.data_ptr(), ol.data_ptr(), ol.stride(0), ll.data_ptr(), T, Hq, Hk, D, 0,
                                          Hq * D, (Hq + Hk) * D, meta.tiles_bwd.data_ptr(), meta.n_tiles, dqkv.data_ptr(), dqkv.stride(0),
                                          acc.data_ptr(), delta.data_ptr(), D ** -0.5, word, st)
        else:
            rc = lib.axb_flash_varlen_bwd_cp(ql.data_ptr(), ql.stride(0), n, off, kv.data_ptr(), kv.stride(0), T, dl.data_ptr(), ol.data_ptr(),
                                             ol.stride(0), ll.data_ptr(), Hq, Hk, D, meta.tiles_bwd.data_ptr(), meta.n_tiles, dqkv.data_ptr(),
                                             dqkv.stride(0), acc.data_ptr(), delta.data_ptr(), D ** -0.5, 1, T, None, word, st)
        _lib.check_rc(rc, "bwd")
        got, ref = dqkv[:n, :Hq * D].float(), want[off:off + n, :Hq * D]
        _lib.check_status()
        assert (acc[n * Hq * D:] == 5.0).all()
        assert ((got - ref).abs() <= 2 ** -6 * want[:, :Hq * D].abs().max()).all()


@pytest.mark.parametrize("lens", [[3], [17], [1, 130], [2, 131, 64], [3, 97, 35]])
@pytest.mark.parametrize("window", [0, 20])
def test_wide_attention_gradient_by_row_alignment(lens, window):
    """256-wide heads: documents that begin at every place of a group of four rows of the dQ sums, tiles that end inside 16 queries, masked
    and unmasked tiles; tolerances of test_attention_head_and_token_remainders."""
    torch.manual_seed(sum(lens))
    D, Hq, Hk, T = 256, 4, 2, sum(lens)
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda").bfloat16().requires_grad_(True)
    do = torch.randn(T, Hq * D, device="cuda").bfloat16()
    meta = Fn.AttnMeta(np.concatenate([[0], np.cumsum(lens)]), "cuda")
    meta = meta.windowed(window) if window else meta
    (g,) = torch.autograd.grad(Fn.flash_varlen(qkv, meta, Hq, Hk, D), qkv, do)
    x = qkv.detach().float().requires_grad_(True)
    q, k, v = (t.reshape(T, -1, D) for t in x.split([Hq * D, Hk * D, Hk * D], -1))
    (want,) = torch.autograd.grad(Fn._attn_ref(q, k, v, meta.cu_seqlens_host, D ** -0.5, True, window).reshape(T, -1), x, do.float())
    _lib.check_status()
    assert ((g.float() - want).abs() <= 2 ** -6 * want.abs().max()).all()
    assert ((g.float() - want).norm() / want.norm()).item() < 2 ** -7


@pytest.mark.parametrize("T,nh,D,rot", [(1, 1, 64, 64), (3, 5, 128, 128), (9, 40, 128, 128), (700, 36, 64, 64), (2500, 10, 256, 128)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_rope_head_groups(T, nh, D, rot, sign):
    """Head counts around the groups of four, few and many tokens (heads over blockIdx.y or not), partial rotation, a row
    stride of its own; the columns behind the heads stay untouched. One bf16 rounding of an fp32 rotation; the angle's own
    rounding (2^-24 of up to T radians) is far below it."""
    torch.manual_seed(T + nh)
    buf = torch.randn(T, nh * D + 24, device="cuda").bfloat16()
    want = buf.clone()
    pos = torch.randint(0, max(2, T), (T,), dtype=torch.int32, device="cuda")
    inv = 1.0 / (10000.0 ** (torch.arange(0, rot, 2, device="cuda").float() / rot))
    _lib.check_rc(_lib.cuda_lib().axb_rope_partial(buf.data_ptr(), pos.data_ptr(), inv.data_ptr(), T, nh, D, rot, buf.stride(0), sign, 1.0,
                                                   _lib.stream_ptr()), "rope_partial")
    x = want[:, :nh * D].reshape(T, nh, D).double()
    ang = (pos.float()[:, None, None] * inv).double()
    a, b = x[..., :rot // 2], x[..., rot // 2:rot]
    r = torch.cat([a * ang.cos() - sign * b * ang.sin(), b * ang.cos() + sign * a * ang.sin(), x[..., rot:]], -1).reshape(T, -1)
    assert ((buf[:, :nh * D].double() - r).abs() <= 2 ** -8 * r.abs() + 2 ** -12).all()
    assert torch.equal(buf[:, nh * D:], want[:, nh * D:])


@pytest.mark.parametrize("V", [5, 264, 8192 + 3, 40960, 40968, 65536 + 7, 128256])
@pytest.mark.parametrize("cap", [0.0, 5.0])
def test_ce_row_edges(V, cap):
    """Both block sizes, tails behind the last vector and partly filled groups of vectors, rows with -inf (masked) logits, an
    ignored row, the label at either end. The gradient is one bf16 rounding of an fp32 softmax whose exponent (up to ~20, exp
    within 2^-21) and sum carry below 2^-12."""
    torch.manual_seed(V)
    R, ld = 6, (V + 7) // 8 * 8 + 8
    z = torch.randn(R, ld, device="cuda").mul_(4).bfloat16()
    z[0, : V // 2] = float("-inf") if not cap else -1e4
    z[1, 1:V] = float("-inf") if not cap else -1e4      # one finite logit
    lab = torch.tensor([V - 1, 0, -100, V // 2, V - 1, 0], device="cuda")
    want = z.clone()
    loss, lse = torch.empty(2, R, device="cuda")
    args = (z.data_ptr(), lab.data_ptr(), loss.data_ptr(), lse.data_ptr(), R, V, ld, 0.5, -100, 1)
    lib = _lib.cuda_lib()
    _lib.check_rc(lib.axb_ce_fwd_bwd_softcap(*args, cap, _lib.stream_ptr()) if cap else lib.axb_ce_fwd_bwd(*args, _lib.stream_ptr()), "ce")
    x = want[:, :V].double()
    t = torch.tanh(x / cap) if cap else x
    e = cap * t if cap else x
    ref_lse = torch.logsumexp(e, -1)
    g = torch.exp(e - ref_lse[:, None])
    keep = lab != -100
    idx = lab.clamp_min(0)
    g[torch.arange(R), idx] -= 1.0
    if cap:
        g = g * (1 - t * t)
    g = torch.where(keep[:, None], 0.5 * g, torch.zeros_like(g))
    assert ((lse - ref_lse).abs() <= 2 ** -19 * (1 + ref_lse.abs())).all()
    ref_loss = torch.where(keep, ref_lse - e[torch.arange(R), idx], torch.zeros_like(ref_lse))
    assert ((loss - ref_loss).abs() <= 2 ** -18 * (1 + ref_lse.abs())).all()
    assert ((z[:, :V].double() - g).abs() <= (2 ** -8 + 2 ** -12) * g.abs() + 2 ** -20).all()
    assert torch.equal(z[:, V:], want[:, V:])


@pytest.mark.parametrize("V", [5, 264, 8192 + 3, 40960, 40968, 128256])
def test_capped_ce_counts_masked_logits(V):
    """cap * tanh(-inf) = -cap is an ordinary term of the sum: all logits -inf but one (at either end, so that the groups
    before and behind a finite one hold nothing else), all of them, and a masked label. Bounds as in ``test_ce_row_edges``."""
    cap, R, ld = 5.0, 4, (V + 7) // 8 * 8
    z = torch.full((R, ld), float("-inf"), device="cuda").bfloat16()
    z[0, 0], z[1, V - 1], z[3, V // 2] = 1.0, 1.0, 7.0
    lab = torch.tensor([0, V - 1, V // 2, 0], device="cuda")
    x = z[:, :V].double()
    loss, lse = torch.empty(2, R, device="cuda")
    _lib.check_rc(_lib.cuda_lib().axb_ce_fwd_bwd_softcap(z.data_ptr(), lab.data_ptr(), loss.data_ptr(), lse.data_ptr(), R, V, ld, 0.5, -100, 1,
                                                         cap, _lib.stream_ptr()), "ce")
    t = torch.tanh(x / cap)
    ref_lse = torch.logsumexp(cap * t, -1)
    g = torch.exp(cap * t - ref_lse[:, None])
    ref_loss = ref_lse - cap * t[torch.arange(R), lab]
    g[torch.arange(R), lab] -= 1.0
    g = 0.5 * g * (1 - t * t)
    assert ((lse - ref_lse).abs() <= 2 ** -19 * (1 + ref_lse.abs())).all()
    assert ((loss - ref_loss).abs() <= 2 ** -18 * (1 + ref_lse.abs())).all()
    assert ((z[:, :V].double() - g).abs() <= (2 ** -8 + 2 ** -12) * g.abs() + 2 ** -20).all()


@pytest.mark.parametrize("D,Dv", [(64, 64), (128, 128), (256, 256), (192, 128)])
@pytest.mark.parametrize("scale", [1.0, 3.0])
@pytest.mark.parametrize("docs", [[0, 1, 130, 1100], [0, 640]])
def test_attention_output_is_rounded_like_a_maximum_referenced_softmax(D, Dv, scale, docs):
    """Rising row maxima over several key blocks (every block of the ring, O rescaled), flat and peaked rows. P is rounded to
    bf16 against the row's own maximum so far: the error is at most that of P (2^-9 relative, its root mean square 2^-9 /
    sqrt(3) with the largest P exact) and of the output (the same), 2^-9 together; 1.15 for the spread."""
    from axolotl_b200.ops import functional as Fn

    torch.manual_seed(D)
    T, Hq, Hk = docs[-1], 4, 2
    qkv = torch.randn(T, Hq * D + Hk * (D + Dv), device="cuda")
    qkv[:, : (Hq + Hk) * D] *= scale
    qkv = qkv.bfloat16()
    out = Fn.flash_varlen(qkv, Fn.AttnMeta(docs, "cuda"), Hq, Hk, D, Dv=Dv)
    _lib.check_status()
    q, k, v = (t.double() for t in qkv.split([Hq * D, Hk * D, Hk * Dv], 1))
    ref = torch.empty(T, Hq, Dv, dtype=torch.double, device="cuda")
    for a, b in zip(docs, docs[1:]):
        for h in range(Hq):
            g = h // (Hq // Hk)
            s = q[a:b, h * D:(h + 1) * D] @ k[a:b, g * D:(g + 1) * D].t() / D ** 0.5
            s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
            ref[a:b, h] = torch.softmax(s, -1) @ v[a:b, g * Dv:(g + 1) * Dv]
    assert (out.double().view_as(ref) - ref).norm() <= 1.15 * 2 ** -9 * ref.norm()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_windowed_attention_does_not_touch_blocks_outside_the_window(D, bad):
    """Heads that pair neighbouring q tiles: a non-finite value row reaches the q tiles whose window includes its key block and no
    other one. The other rows are those of a clean run, bit for bit."""
    from axolotl_b200.ops import functional as Fn

    torch.manual_seed(D)
    T, H, win = 4096, 8, 64
    qkv = torch.randn(T, 3 * H * D, device="cuda").bfloat16()
    meta = Fn.AttnMeta([0, T], "cuda").windowed(win)
    clean = Fn.flash_varlen(qkv, meta, H, H, D)
    qkv[200, 2 * H * D:] = bad
    out = Fn.flash_varlen(qkv, meta, H, H, D)
    _lib.check_status()
    far = torch.ones(T, dtype=torch.bool, device="cuda")
    far[128:384] = False
    assert torch.equal(out[far], clean[far]) and torch.isfinite(clean).all()
