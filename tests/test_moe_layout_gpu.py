"""Layout of a routed batch, dispatch and combine kernels against plain PyTorch."""
import pytest
import torch

from axolotl_b200.ops import _lib
from axolotl_b200.ops.grouped import BLOCK, GroupLayout, RoutedLayout, grouped_gemm, grouped_gemm_w4a16
from axolotl_b200.ops.nvfp4 import dequantize_nvfp4, quantize_nvfp4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (3, 2, 8), (333, 8, 128), (128, 8, 8), (1025, 1, 5), (700, 6, 160), (200, 4, 1024), (40, 2, 1500)])
@pytest.mark.parametrize("skew", [False, True])
def test_routed_layout(T, k, E, skew):
    """Slot counts at the edges of the 1024-slot blocks and of warps, experts without slots, one expert with all of them,
    expert counts at and above the placing kernel's threads: the layout of a stable sort, exactly."""
    from axolotl_b200.ops.grouped import BLOCK, RoutedLayout

    torch.manual_seed(T + E)
    idx = torch.stack([torch.randperm(E)[:k] if E >= k else torch.zeros(k, dtype=torch.long) for _ in range(T)])
    if skew:
        idx = (idx * 0 + E - 1) if E < 8 else idx % max(1, E // 4)
    lay = RoutedLayout(idx.cuda(), E)
    flat = idx.reshape(-1)
    counts = torch.bincount(flat, minlength=E)
    padded = (counts + BLOCK - 1) // BLOCK * BLOCK
    start = padded.cumsum(0) - padded
    order = torch.argsort(flat, stable=True)
    dest = torch.cat([torch.arange(int(c)) + int(s) for c, s in zip(counts, start)])
    slot_row = torch.empty(T * k, dtype=torch.long)
    slot_row[order] = dest
    row_slot = torch.full((lay.max_rows,), -1, dtype=torch.long)
    row_slot[dest] = order
    nb = int(padded.sum()) // BLOCK
    assert int(lay.n_blocks) == nb and lay.max_rows >= nb * BLOCK
    assert torch.equal(lay.slot_row.long().cpu(), slot_row) and torch.equal(lay.row_slot.long().cpu(), row_slot)
    assert torch.equal(lay.seg_rows.long().cpu(), padded) and torch.equal(lay.seg_start.long().cpu(), start)
    blk = torch.searchsorted(padded.cumsum(0), torch.arange(lay.max_blocks) * BLOCK, right=True).clamp(max=E - 1)
    assert torch.equal(lay.blk_expert.long().cpu(), blk)


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (333, 8, 128), (40, 2, 1500)])
def test_routed_layout_pads_and_unpads(T, k, E):
    """The compact form of a routed batch (slots in expert order) through the padded layout and back, exactly."""
    from axolotl_b200.ops.grouped import RoutedLayout

    idx = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).cuda()
    lay = RoutedLayout(idx, E)
    x = torch.randn(T * k, 16, device="cuda").bfloat16()
    order = torch.argsort(idx.reshape(-1), stable=True)
    p = lay.pad(x[order])
    assert torch.equal(lay.unpad(p), x[order]) and torch.equal(p[lay.slot_row.long()], x)
    assert int((p != 0).any(1).sum()) == T * k


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (5, 3, 256), (37, 8, 2048), (19, 9, 2056), (3, 16, 264)])
def test_dispatch_and_combine_rows(T, k, H):
    """Widths around the 256-column chunks and eight vectors in flight, more than eight slots per token. One bf16 rounding of
    an fp32 sum (2^-8); the weight gradient is an fp32 dot product (2^-18 of its magnitude)."""
    from axolotl_b200.ops.grouped import RoutedLayout, _combine_rows, _dispatch_rows

    torch.manual_seed(T + H)
    E = 16
    idx = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).cuda()
    lay = RoutedLayout(idx, E)
    x, w = torch.randn(T, H, device="cuda").bfloat16(), torch.rand(T, k, device="cuda")
    rows = lay.row_slot.long()
    live = rows >= 0
    for scale in (None, w):
        out = _dispatch_rows(x, lay, scale)
        ref = x[rows.clamp(min=0) // k].float() * (scale.reshape(-1)[rows.clamp(min=0)][:, None] if scale is not None else 1.0)
        assert torch.equal(out, torch.where(live[:, None], ref.bfloat16(), torch.zeros_like(out)))
    ys = torch.randn(lay.max_rows, H, device="cuda").bfloat16()
    for scale in (None, w):
        out = _combine_rows(ys, lay.slot_row, scale, T, k)
        ref = (ys[lay.slot_row.long()].view(T, k, H).double() * (scale.double()[..., None] if scale is not None else 1.0)).sum(1)
        assert ((out.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()
    dw = torch.empty(T, k, device="cuda")
    dy = torch.randn(T, H, device="cuda").bfloat16()
    _lib.check_rc(_lib.cuda_lib().axb_moe_combine_dw(dy.data_ptr(), ys.data_ptr(), lay.slot_row.data_ptr(), dw.data_ptr(), T * k, k, H,
                                                     _lib.stream_ptr()), "moe_combine_dw")
    prod = dy.double()[:, None] * ys[lay.slot_row.long()].view(T, k, H).double()
    assert ((dw.double() - prod.sum(-1)).abs() <= 2 ** -18 * prod.abs().sum(-1)).all()


def test_slots_of_experts_that_do_not_exist():
    """They get no row, the others keep theirs; combination and weight gradient take them for zero and the status word tells."""
    from axolotl_b200.ops.grouped import RoutedLayout, _combine_rows

    torch.manual_seed(0)
    T, k, E, H = 700, 3, 8, 64
    idx = torch.randint(0, E, (T, k), device="cuda")
    clean = RoutedLayout(torch.where(idx == 5, 4, idx), E)      # an expert without rows of its own
    bad = idx == 5
    idx = torch.where(bad, torch.tensor([E, -1, 2 ** 40], device="cuda")[torch.arange(k, device="cuda")].expand(T, k), idx)
    lay = RoutedLayout(idx, E)
    with pytest.raises(_lib.KernelBoundsError):
        _lib.check_status()
    flat = bad.reshape(-1)
    assert (lay.slot_row[flat] == -1).all() and (lay.slot_row[~flat] >= 0).all()
    live = lay.row_slot >= 0
    assert int(live.sum()) == int((~flat).sum())
    assert torch.equal(lay.slot_row[lay.row_slot[live].long()].long(), live.nonzero().squeeze(1))
    assert torch.equal(lay.seg_rows[[0, 1, 2, 3, 6, 7]], clean.seg_rows[[0, 1, 2, 3, 6, 7]]) and lay.seg_rows[5] == 0
    ys, w = torch.randn(lay.max_rows, H, device="cuda").bfloat16(), torch.rand(T, k, device="cuda")
    rows = ys[lay.slot_row.clamp(min=0).long()].view(T, k, H).double() * (~bad)[..., None]
    out = _combine_rows(ys, lay.slot_row, w.masked_fill(bad, float("nan")), T, k)
    ref = (rows * w.double()[..., None]).sum(1)
    assert ((out.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()
    dw, dy = torch.empty(T, k, device="cuda"), torch.randn(T, H, device="cuda").bfloat16()
    _lib.check_rc(_lib.cuda_lib().axb_moe_combine_dw(dy.data_ptr(), ys.data_ptr(), lay.slot_row.data_ptr(), dw.data_ptr(), T * k, k, H,
                                                     _lib.stream_ptr()), "moe_combine_dw")
    prod = dy.double()[:, None] * rows
    assert ((dw.double() - prod.sum(-1)).abs() <= 2 ** -18 * prod.abs().sum(-1)).all()


@pytest.mark.parametrize("R,C", [(1, 1), (63, 65), (64, 64), (130, 7), (8, 24576), (4099, 128)])
def test_transpose_modes(R, C):
    """Tile edges; the bf16 form is one rounding, the fp32 forms are exact."""
    from axolotl_b200.ops import _lib

    a = torch.randn(R, C, device="cuda")
    base = torch.randn(C, R, device="cuda")
    for mode, dst, want in ((0, torch.empty(C, R, device="cuda", dtype=torch.bfloat16), a.t().bfloat16()),
                            (1, base.clone(), base + a.t()), (2, torch.empty(C, R, device="cuda"), a.t())):
        _lib.check_rc(_lib.cuda_lib().axb_transpose(a.data_ptr(), dst.data_ptr(), R, C, mode, _lib.stream_ptr()), "transpose")
        assert torch.equal(dst, want)


@pytest.mark.parametrize("counts", [[1, 31, 32, 33, 0, 127, 128, 129], [255, 256, 257, 0, 385], [0, 3], [700]])
def test_passes_of_a_routed_layout(counts):
    """Every row block is in one pass of its expert; the table that the placing kernel writes holds the passes that the general one
    gives, with the rows in use instead of whole blocks."""
    E, T = len(counts), sum(counts)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T)].view(T, 1).cuda()
    lay = RoutedLayout(idx, E)
    got, n = lay.passes[0].cpu(), int(lay.passes[1])
    ref, n_ref = GroupLayout.passes.func(lay)
    assert n == int(n_ref) == sum(-(-c // 256) for c in counts)
    assert torch.equal(got[:n, [0, 1, 3]], ref.cpu()[:n, [0, 1, 3]])
    assert got[:n, 2].tolist() == [min(256, c - a) for c in counts for a in range(0, c, 256)]


@pytest.mark.parametrize("N,K,r", [(8, 64, 0), (136, 64, 16), (264, 192, 8), (512, 320, 16)])
def test_grouped_w4a16_rows_in_use(N, K, r):
    """Passes of few rows, short sums (fewer k blocks than converter groups), columns that end inside a tile and negative block scales:
    the bits of the bf16 stack in the grouped GEMM, and zeros in the rows that pad a segment."""
    counts = [1, 31, 0, 33, 129, 255, 257, 64, 0, 128]
    E, T = len(counts), sum(counts)
    torch.manual_seed(N)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).view(T, 1).cuda()
    lay = RoutedLayout(idx, E)
    qd, sc, pts = quantize_nvfp4(torch.randn(E, N, K) * 0.05)
    sc = (sc.float() * torch.where(torch.rand(sc.shape) < 0.1, -1.0, 1.0)).to(sc.dtype)
    q = {"qdata": qd.cuda(), "scale": sc.cuda(), "pts": pts.cuda()}
    W = dequantize_nvfp4(q["qdata"], q["scale"], q["pts"])
    pad = lambda c, s=0.5: torch.where(lay.row_slot[:, None] >= 0, torch.randn(lay.max_rows, c, device="cuda") * s, 0.0).bfloat16()  # noqa: E731
    x, dy, t = pad(K), pad(N), pad(max(r, 8))
    A16, Bt = (torch.randn(E, r, K, device="cuda") * 0.05).bfloat16(), (torch.randn(E, N, r, device="cuda") * 0.05).bfloat16()
    ext = lambda w: dict(a2=t[:, :r].contiguous(), w2=w) if r else {}  # noqa: E731
    used = int(lay.n_blocks) * BLOCK
    empty = lay.row_slot[:used] < 0
    for got, ref in ((grouped_gemm_w4a16(x, q, lay, **ext(Bt)), grouped_gemm(x, W, lay, **ext(Bt))),
                     (grouped_gemm_w4a16(dy, q, lay, trans_w=True, **ext(A16)), grouped_gemm(dy, W, lay, trans_w=True, **ext(A16)))):
        _lib.check_status()
        assert torch.equal(got[:used], ref[:used]) and not got[:used][empty].any()
    y32 = grouped_gemm_w4a16(x, q, lay, out_dtype=torch.float32)[:used]
    assert torch.equal(y32.bfloat16(), grouped_gemm(x, W, lay)[:used])


def test_grouped_w4a16_repeats_its_bits_under_load():
    """Several passes on every SM pair, k blocks of every ring position, the LoRA extension and full, half and nearly empty passes side
    by side, twenty times: a tile that the tensor core read before the other CTA's part of it was in place would change some bit."""
    E, N, K, r = 48, 1536, 2048, 16
    counts = [(37 * e) % 600 for e in range(E)]
    torch.manual_seed(5)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).view(-1, 1).cuda()
    lay = RoutedLayout(idx, E)
    q = dict(zip(("qdata", "scale", "pts"), (t.cuda() for t in quantize_nvfp4(torch.randn(E, N, K) * 0.05))))
    W = dequantize_nvfp4(q["qdata"], q["scale"], q["pts"])
    pad = lambda c: torch.where(lay.row_slot[:, None] >= 0, torch.randn(lay.max_rows, c, device="cuda"), 0.0).bfloat16()  # noqa: E731
    x, dy, t = pad(K), pad(N), pad(r)
    A16, Bt = torch.randn(E, r, K, device="cuda").bfloat16(), torch.randn(E, N, r, device="cuda").bfloat16()
    used = int(lay.n_blocks) * BLOCK
    for a, w2, tr in ((x, Bt, False), (dy, A16, True)):
        want = grouped_gemm(a, W, lay, trans_w=tr, a2=t, w2=w2)[:used]
        for _ in range(20):
            assert torch.equal(grouped_gemm_w4a16(a, q, lay, trans_w=tr, a2=t, w2=w2)[:used], want)
    _lib.check_status()


def _passes(counts, max_blocks):
    out, b = [], 0
    for e, c in enumerate(counts):
        nb = -(-c // BLOCK)
        out += [[b + j, e, min(c - j * BLOCK, 256, (max_blocks - b - j) * BLOCK), min(2, nb - j, max_blocks - b - j)]
                for j in range(0, nb, 2) if b + j < max_blocks]
        b += nb
    return out


@pytest.mark.parametrize("counts", [[1, 31, 32, 33, 0, 127, 128, 129], [255, 256, 257, 0, 385], [0], [0, 3], [700],
                                    [(7 * e) % 300 for e in range(1025)], [0] * 1024 + [5, 0, 400] + [1] * 1100])
def test_passes_of_a_layout_by_counts(counts):
    """The layouts of the expert-parallel and the general path know their rows too: rows in use, not whole blocks, for any number of
    experts."""
    lay = GroupLayout(torch.tensor(counts, device="cuda"), sum(counts))
    table, n = lay.passes
    assert table.shape == (lay.max_blocks, 4) and table[: int(n)].tolist() == _passes(counts, lay.max_blocks)


@pytest.mark.parametrize("cf", [0.25, 0.6, 4.0])
def test_passes_of_an_expert_parallel_plan(cf):
    """The plan that is made on the device, with room for all rows and with too little of it (more rows than the capacity: reported, and
    the segments end at the last block): every pass inside the blocks that exist."""
    from axolotl_b200.parallel.ep import ExpertParallelGroup

    world, E, T, k = 4, 16, 512, 2
    torch.manual_seed(3)
    g = ExpertParallelGroup.__new__(ExpertParallelGroup)
    g.device, g.size, g.rank, g.E, g.E_local = torch.device("cuda"), world, 0, E, E // world
    g.fused, g.dedup, g.overflow, g.capacity_factor = False, True, None, cf
    all_idx = torch.randint(0, 6, (world * T * k,), dtype=torch.int32, device="cuda")      # mostly this rank's experts
    lay = g._plan_from_tables(all_idx, torch.ones(world * T * k, device="cuda"), all_idx[: T * k].reshape(T, k), 8).lay
    counts = [int((all_idx == e).sum()) for e in range(E // world)]
    want = _passes(counts, lay.max_blocks)
    assert bool(g.overflow) == (cf < 2) and int(lay.n_blocks) == sum(p[3] for p in want)
    assert lay.passes[0][: int(lay.passes[1])].tolist() == want


def test_rows_in_use_of_a_general_layout():
    """NVFP4 experts over segments given by their counts, short ones among them: the bits of the bf16 stack, zeros in the padding."""
    counts, N, K = [1, 31, 0, 33, 129, 255, 257, 64, 0, 128], 136, 192
    torch.manual_seed(7)
    lay = GroupLayout(torch.tensor(counts, device="cuda"), sum(counts))
    q = dict(zip(("qdata", "scale", "pts"), (t.cuda() for t in quantize_nvfp4(torch.randn(len(counts), N, K) * 0.05))))
    W = dequantize_nvfp4(q["qdata"], q["scale"], q["pts"])
    used = int(lay.n_blocks) * BLOCK
    for a, tr in ((lay.pad(torch.randn(sum(counts), K, device="cuda").bfloat16()), False),
                  (lay.pad(torch.randn(sum(counts), N, device="cuda").bfloat16()), True)):
        assert torch.equal(grouped_gemm_w4a16(a, q, lay, trans_w=tr)[:used], grouped_gemm(a, W, lay, trans_w=tr)[:used])
    _lib.check_status()
