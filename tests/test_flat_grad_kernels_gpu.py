"""Flat fp32 gradient buffers: embedding and loss-head gradients added in place, square sum, AdamW."""
import math

import pytest
import torch

from axolotl_b200.ops import _lib
from axolotl_b200.ops import functional as Fn
from axolotl_b200.ops.optim import adamw_step_, grad_sumsq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 2048, 1036, 33])
@pytest.mark.parametrize("off", [0, 1])
def test_embedding_bwd_forms(H, off):
    """16-byte and element form (width or table off the grid), ids of a ragged batch with repeats. fp32 sums in any order."""
    torch.manual_seed(H)
    T, V = 301, 50
    d = torch.randn(T, H, device="cuda").bfloat16()
    ids = torch.randint(0, V, (T,), device="cuda")
    buf = torch.randn(V * H + off + 3, device="cuda")
    tab = buf[off:off + V * H].view(V, H)
    ref = tab.double().index_add(0, ids, d.double())
    mag = tab.double().abs().index_add(0, ids, d.double().abs())
    rest = buf[off + V * H:].clone()
    _lib.check_rc(_lib.cuda_lib().axb_embedding_bwd(d.data_ptr(), ids.data_ptr(), tab.data_ptr(), T, H, V, _lib.stream_ptr()), "embedding_bwd")
    assert ((tab.double() - ref).abs() <= 2 ** -20 * mag).all() and torch.equal(buf[off + V * H:], rest)


@pytest.mark.parametrize("n", [1, 3, 1024, 5_000_003])
@pytest.mark.parametrize("off", [0, 1])
def test_flat_sumsq_axpy_adamw(n, off):
    """Vector body and element tail, aligned and not. n terms summed by at most 2^13 steps per lane: 2^-12 for the sum."""
    torch.manual_seed(n)
    big = torch.randn(4, n + off, device="cuda")
    flat = [torch.empty(n + off, device="cuda").copy_(b)[off:] for b in big]
    p, g, m, v = flat
    v.abs_()
    ss = grad_sumsq(g, None)
    assert math.isclose(float(ss), float(g.double().pow(2).sum()), rel_tol=2 ** -12)
    y, want = torch.randn(n + off, device="cuda")[off:], None
    want = y.double() + 0.75 * g.double()
    _lib.check_rc(_lib.cuda_lib().axb_axpy_f32(y.data_ptr(), g.data_ptr(), torch.full((), 0.75, device="cuda").data_ptr(), n,
                                               _lib.stream_ptr()), "axpy")
    assert ((y.double() - want).abs() <= 2 ** -23 * (want.abs() + g.abs())).all()
    lr, b1, b2, eps, wd, step = 1e-2, 0.9, 0.95, 1e-6, 0.1, 3
    P, G, M, W = (t.double() for t in (p, g, m, v))
    M = b1 * M + (1 - b1) * G
    W = b2 * W + (1 - b2) * G * G
    upd = lr * (M / (1 - b1 ** step)) / ((W / (1 - b2 ** step)).sqrt() + eps)
    ref = P * (1 - lr * wd) - upd
    copy = torch.empty(n + off, device="cuda", dtype=torch.bfloat16)[off:]
    adamw_step_(p, g, m, v, lr=lr, beta1=b1, beta2=b2, eps=eps, weight_decay=wd, step=step, bf16_copy=copy)
    # a handful of fp32 roundings (1 - beta in fp32: 2^-24 / 0.05) of operands of these magnitudes
    assert ((p.double() - ref).abs() <= 2 ** -19 * (P.abs() + upd.abs() + lr)).all()
    assert torch.equal(copy, p.bfloat16())


@pytest.mark.parametrize("T,V", [(64, 512), (640, 4096)])
def test_head_and_table_gradients_reach_the_flat_buffer(T, V):
    """With an optimizer buffer the gradients are added to it (twice here, two chunks), without one they come back rounded to bf16."""
    torch.manual_seed(T)
    H = 256
    ids, labels = torch.randint(0, V, (2, T), device="cuda")
    tab0, w0 = (torch.randn(V, H, device="cuda") * 0.1).bfloat16(), (torch.randn(V, H, device="cuda") * 0.1).bfloat16()
    def run(flat):
        tab, w = torch.nn.Parameter(tab0.clone()), torch.nn.Parameter(w0.clone())
        if flat:
            tab._axb_grad, w._axb_grad = torch.ones(2, V, H, device="cuda")
        for _ in range(2 if flat else 1):
            (Fn.linear_cross_entropy(Fn.embedding(tab, ids), w, labels, chunk_rows=T // 2) * 3.0).backward()
        if flat:
            assert tab.grad is None and w.grad is None
            return tab._axb_grad.sub(1).div(2), w._axb_grad.sub(1).div(2)
        return tab.grad.float(), w.grad.float()
    for a, b in zip(run(True), run(False)):
        # one bf16 rounding of the returned gradient; the buffer's ones cost 2^-23 of themselves per addition
        assert ((a - b).abs() <= 2 ** -8 * b.abs() + 2 ** -20).all()


def _loss(tab, w, ids, labels):
    return Fn.linear_cross_entropy(Fn.embedding(tab, ids), w, labels)


@pytest.mark.parametrize("kind", ["hook", "post", "grad", "inputs", "partial"])
def test_flat_buffer_leaves_hooks_and_partial_backwards_alone(kind):
    """Hooks on the table or the head see (and may change) their gradient, ``torch.autograd.grad`` returns it, and a backward pass
    restricted to other inputs adds nothing to the buffers."""
    torch.manual_seed(0)
    V, H, T = 512, 256, 64
    ids, labels = torch.randint(0, V, (2, T), device="cuda")
    tab, w = (torch.nn.Parameter((torch.randn(V, H, device="cuda") * 0.1).bfloat16()) for _ in range(2))
    want = torch.autograd.grad(_loss(tab, w, ids, labels), (tab, w))
    for p in (tab, w):
        p._axb_grad = torch.zeros(V, H, device="cuda")
    seen = []
    if kind == "hook":
        for p in (tab, w):
            p.register_hook(lambda g: seen.append(g) or g * 2)
        _loss(tab, w, ids, labels).backward()
        assert len(seen) == 2
        got = tab.grad / 2, w.grad / 2
    elif kind == "post":
        for p in (tab, w):
            p.register_post_accumulate_grad_hook(lambda q: seen.append(q.grad))
        _loss(tab, w, ids, labels).backward()
        assert len(seen) == 2
        got = tab.grad, w.grad
    elif kind == "grad":
        got = torch.autograd.grad(_loss(tab, w, ids, labels), (tab, w))
    elif kind == "inputs":
        _loss(tab, w, ids, labels).backward(inputs=[tab])
        assert not w._axb_grad.any() and w.grad is None
        got = tab._axb_grad.bfloat16(), want[1]
        tab._axb_grad.zero_()
    else:
        h = Fn.embedding(tab, ids).detach().requires_grad_(True)
        torch.autograd.grad(Fn.linear_cross_entropy(h, w, labels), h)
        got = want
    assert not tab._axb_grad.any() and not w._axb_grad.any()
    for a, b in zip(got, want):
        assert (a.float() - b.float()).norm() <= 2 ** -7 * b.float().norm()


@pytest.mark.parametrize("M,N,K", [(8, 8, 64), (264, 24, 200), (136, 72, 520), (520, 264, 328), (2056, 1040, 136)])
@pytest.mark.parametrize("bn,splits", [(None, 1), (64, 1), (128, 1), (256, 1), (64, 5), (128, 3)])
@pytest.mark.parametrize("col", [0, 4, 3])
def test_product_added_to_an_fp32_slice(M, N, K, bn, splits, col):
    """dW += dY^T X into columns of a wider buffer, rows and columns that end inside a 32 x 32 tile, aligned slices (tile reductions) and one
    that is not (added from registers): fp32 sums of bf16 products, in another order; the columns beside the slice stay as they are."""
    from axolotl_b200.ops.gemm import gemm

    torch.manual_seed(M + K)
    a, b = torch.randn(K, M, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    buf = torch.randn(M, N + 24, device="cuda")
    old = buf.clone()
    gemm(a, b, trans_a=True, trans_b=True, out=buf[:, col:col + N], accumulate=True, splits=splits, bn=bn, alpha=0.5)
    _lib.check_status()
    want = old.double()
    want[:, col:col + N] += 0.5 * a.double().t() @ b.double()
    size = old.double().abs()
    size[:, col:col + N] += 0.5 * a.double().abs().t() @ b.double().abs()
    assert ((buf.double() - want).abs() <= 2 ** -20 * size).all()
    assert torch.equal(buf[:, :col], old[:, :col]) and torch.equal(buf[:, col + N:], old[:, col + N:])


@pytest.mark.parametrize("M,N,K,bn", [(136, 72, 64, 64), (136, 168, 64, 128), (72, 264, 128, 256), (2056, 2312, 64, 256)])
@pytest.mark.parametrize("col,cin_col", [(3, None), (3, 0), (0, 5), (1, 2), (0, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_results_and_operands_off_16_bytes(M, N, K, bn, col, cin_col, dtype):
    """C and the operand that is added, each on and off a 16-byte boundary while its rows are whole vectors apart, in the single-CTA
    kernel at its three widths and in the pair kernel: one rounding of an fp32 sum of K products, and the columns beside C stay as they
    are."""
    from axolotl_b200.ops import gemm as G

    assert G._use_pair(M, N, bn) == (M > 1000)
    torch.manual_seed(M + col)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    buf, add = torch.randn(M, N + 24, device="cuda").to(dtype), torch.randn(M, N + 24, device="cuda").to(dtype)
    old = buf.clone()
    c_in = None if cin_col is None else add[:, cin_col:cin_col + N]
    G.gemm(a, b, out=buf[:, col:col + N], out_dtype=dtype, c_in=c_in, beta=0.0 if c_in is None else 0.75, alpha=0.5, bn=bn)
    _lib.check_status()
    want, size = 0.5 * a.double() @ b.double().t(), 0.5 * a.double().abs() @ b.double().abs().t()
    if c_in is not None:
        want, size = want + 0.75 * c_in.double(), size + 0.75 * c_in.double().abs()
    got = buf[:, col:col + N].double()
    assert ((got - want).abs() <= (2 ** -8 if dtype == torch.bfloat16 else 0) * want.abs() + 2 ** -20 * size).all()
    assert torch.equal(buf[:, :col], old[:, :col]) and torch.equal(buf[:, col + N:], old[:, col + N:])
