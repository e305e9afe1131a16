"""The attention output that the backward kernels read 16 bytes at a time, at addresses where that would fault."""
import numpy as np
import pytest
import torch

from axolotl_b200.ops import _lib
from axolotl_b200.ops import functional as Fn


@pytest.mark.parametrize("which", ["out", "dqkv", "dq_acc"])
@pytest.mark.parametrize("entry", ["varlen", "wide"])
def test_backward_entries_refuse_unaligned_buffers(entry, which):
    """Refused (-3) before anything is launched: made-up addresses, no GPU."""
    at = {n: 0x10000000 * (i + 1) for i, n in enumerate(("qkv", "dout", "out", "lse", "tiles", "dqkv", "dq_acc", "delta"))}
    at[which] += 4
    lib, T, Hq, Hk = _lib.cuda_lib(), 64, 4, 2
    if entry == "varlen":
        D, ld = 128, (Hq + 2 * Hk) * 128
        rc = lib.axb_flash_varlen_bwd(at["qkv"], ld, at["dout"], at["out"], Hq * D, at["lse"], T, Hq, Hk, D, 0, Hq * D, (Hq + Hk) * D, at["tiles"],
                                      1, at["dqkv"], ld, at["dq_acc"], at["delta"], 0.1, None, None)
    else:
        D, ld = 256, (Hq + 2 * Hk) * 256
        rc = lib.axb_flash_wide_bwd(at["qkv"], ld, at["dout"], at["out"], Hq * D, at["lse"], T, Hq, Hk, D, D, 0, Hq * D, (Hq + Hk) * D, at["tiles"],
                                    1, at["dqkv"], ld, at["dq_acc"], at["delta"], 0.1, 0.0, None, None)
    assert rc == -3


@pytest.mark.gpu
@pytest.mark.parametrize("D,Dv", [(64, 64), (128, 128), (192, 128), (256, 256)])
@pytest.mark.parametrize("shift", [2, 6])
def test_saved_output_at_any_address(D, Dv, shift):
    """Saved-tensor hooks that bring the output back 4 or 12 bytes off a 16-byte boundary: the same gradients, bit for bit (dK and dV have
    one order of summation; the sums of dQ have not)."""
    torch.manual_seed(D)
    Hq, Hk, lens = 2, 2, [70, 130]
    T = sum(lens)
    meta = Fn.AttnMeta(np.concatenate([[0], np.cumsum(lens)]), "cuda")
    qkv = torch.randn(T, (Hq + Hk) * D + Hk * Dv, device="cuda").bfloat16().requires_grad_(True)
    do = torch.randn(T, Hq * Dv, device="cuda").bfloat16()

    def unpack(t):
        if t.shape != (T, Hq * Dv):
            return t
        buf = torch.empty(t.numel() + shift, dtype=t.dtype, device="cuda")
        return buf[shift:].view(t.shape).copy_(t)

    def grad():
        out = Fn._FlashWide.apply(qkv, meta, Hq, Hk, D, Dv, D ** -0.5, 0.0) if D > 128 else Fn.flash_varlen(qkv, meta, Hq, Hk, D)
        return torch.autograd.grad(out, qkv, do)[0].float()

    want = grad()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        got = grad()
    _lib.check_status()
    assert torch.equal(got[:, Hq * D:], want[:, Hq * D:])
    assert ((got - want).abs() <= 2 ** -8 * want.abs() + 2 ** -16 * want.abs().max()).all()
