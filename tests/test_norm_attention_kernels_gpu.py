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
