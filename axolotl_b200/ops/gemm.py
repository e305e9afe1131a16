"""bf16 GEMM on the tcgen05 kernel (CUDA) with a plain PyTorch path for CPU tensors.

``gemm(a, b)`` computes ``alpha * (op(a) @ op(b)^T + a2 @ b2^T) + beta * c_in`` where
``op(a)`` is ``a`` ([M, K]) or, with ``trans_a``, a matrix stored as [K, M]; likewise
``op(b)`` is ``b`` ([N, K]) or, with ``trans_b``, stored as [K, N]. The optional ``a2``/``b2``
pair is the K-extension that fuses a LoRA update into the same accumulator tile.
"""
from __future__ import annotations

import os

import torch

from . import _lib

_SM = 148
# CTA-pair (cta_group::2, 256x256 tile per SM pair) kernel: the default for large GEMMs;
# AXB_GEMM_PAIR=0 keeps every launch on the single-CTA kernel.
USE_PAIR = os.environ.get("AXB_GEMM_PAIR", "1") != "0"
# GLU folded into the gate|up GEMM epilogue (forward) and the down-projection input-gradient GEMM
# (backward); AXB_GLU_EPILOGUE=0 runs the stand-alone GLU kernels instead.
USE_GLU_EPILOGUE = os.environ.get("AXB_GLU_EPILOGUE", "1") != "0"


# tile width, pair kernel?, rows, tiles at once, microseconds per 64-deep K block, microseconds per tile for bf16 results / fp32
# results / results added to an operand read by the epilogue / results added to the fp32 output by tile reductions (L2 flushed; least
# squares over 7600 drawn products, the last over 138)
_TILES = ((256, True, 256, _SM // 2, 0.336, (2.2, 8.7, 25.8, 5.8)), (256, False, 128, _SM, 0.441, (5.6, 8.6, 24.0, 5.4)),
          (128, False, 128, _SM, 0.292, (2.8, 4.3, 11.8, 2.7)), (64, False, 128, _SM, 0.236, (1.3, 2.1, 5.9, 1.2)))


def _pick_tile(M: int, N: int, k_blocks: int = 64, epilogue: int = 0) -> tuple[int, bool]:
    """(tile width, whether the CTA-pair kernel runs it): the choice with the least waves x time per wave. Mostly the number
    of waves decides, 960 x 32000 by 4096 takes 580 / 304 / 200 / 173 us (10, 4, 2, 1 waves with 64, 128, 256, pair); with a
    short K the epilogue does, which the pair kernel has cheapest in bf16 (TMA stores) and wide tiles have dearest where they read
    and write an operand: 1568 x 88 by 13712 51 / 44 / 42 / 26 us, 1304 x 96 by 3720 added to fp32 46 / 51 / 64 / 70. Within 0.8 % of the best of the four on average, 2.7 % by waves alone.
    Ties go to the wider tile, which reads less."""
    best = None
    for bn, pair, rows, slots, per_k, per_tile in _TILES:
        if (pair and not USE_PAIR) or (bn > 64 and N <= bn // 2) or (pair and (M <= 128 or N < 256)):
            continue
        t = -(-(-(-M // rows) * -(-N // bn)) // slots) * (per_k * k_blocks + per_tile[epilogue])
        if best is None or t < best[0]:
            best = (t, bn, pair)
    return best[1], best[2]


def _row_major_2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        raise ValueError("gemm operands must be 2-D")
    if t.stride(1) != 1 or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
        if t.stride(0) % 8 != 0:
            raise ValueError("gemm operand rows must be a multiple of 8 elements")
    return t


def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    *,
    trans_a: bool = False,
    trans_b: bool = False,
    a2: torch.Tensor | None = None,
    b2: torch.Tensor | None = None,
    alpha: float = 1.0,
    beta: float = 0.0,
    c_in: torch.Tensor | None = None,
    out: torch.Tensor | None = None,
    out_dtype: torch.dtype = torch.bfloat16,
    accumulate: bool = False,
    splits: int = 1,
    bn: int | None = None,
    glu: tuple | None = None,
) -> torch.Tensor:
    """``glu`` selects a GLU epilogue of the CTA-pair kernel (callers check ``glu_fusable`` first):
    ``("fwd", kind, limit, h_out)``: ``b`` is the [2I, K] gate|up weight, ``out`` [M, 2I] receives
    gate|up and ``h_out`` [M, I] ``act(gate) * up``; ``("bwd", kind, limit, gate_up)``: the product is
    dh [M, I] and ``out`` [M, 2I] receives d_gate | d_up (``out`` may be ``gate_up`` itself)."""
    quant = getattr(b, "_axb_quant", None)
    if quant is not None:
        # frozen 4-bit weight: expand into the shared bf16 scratch right before the GEMM reads it
        from .nf4 import dequantize_nf4, scratch_weight

        b = dequantize_nf4(b, quant, out=scratch_weight(quant.shape, b.device) if b.is_cuda else None,
                           dtype=torch.bfloat16 if b.is_cuda else a.dtype)
    shard = getattr(b, "_axb_shard", None)
    if shard is not None:
        return _gemm_allgather(a, b, shard, trans_a=trans_a, trans_b=trans_b, a2=a2, b2=b2, alpha=alpha,
                               beta=beta, c_in=c_in, out=out, out_dtype=out_dtype, bn=bn, glu=glu)
    M, K = (a.shape[1], a.shape[0]) if trans_a else a.shape
    N = b.shape[1] if trans_b else b.shape[0]
    Kb = b.shape[0] if trans_b else b.shape[1]
    if K != Kb:
        raise ValueError(f"gemm: inner dimensions differ ({K} vs {Kb})")
    K2 = 0
    if a2 is not None:
        K2 = a2.shape[0] if trans_a else a2.shape[1]

    if not a.is_cuda:
        # reference path (CPU): same contraction in the operand dtype with fp32 accumulation
        fa = (a.t() if trans_a else a).float()
        fb = (b if trans_b else b.t()).float()
        acc = fa @ fb
        if a2 is not None:
            acc = acc + (a2.t() if trans_a else a2).float() @ (b2 if trans_b else b2.t()).float()
        acc = acc * alpha
        if c_in is not None and beta != 0.0:
            acc = acc + beta * c_in.float()
        if accumulate:
            out.add_(acc.to(out.dtype))
            return out
        res = acc.to(out_dtype if a.dtype == torch.bfloat16 or out_dtype == torch.float32 else a.dtype)
        if out is not None:
            out.copy_(res)
            return out
        return res

    lib = _lib.cuda_lib()
    if a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
        raise TypeError("the tcgen05 GEMM takes bf16 operands")
    a = _row_major_2d(a)
    b = _row_major_2d(b)
    if a2 is not None:
        a2 = _row_major_2d(a2)
        b2 = _row_major_2d(b2)
    if (accumulate and splits > 1 and trans_a and trans_b and M <= 64 and N >= 512 and K >= 256 and a2 is None and c_in is None and glu is None
            and out is not None and out.dtype == torch.float32 and out.stride(1) == 1):
        # dA = t^T x of an adapter: the long side goes to the 128-row operand (with t there, 128 - M rows of every tile are
        # padding and the tile reads three times the bytes) and the epilogue adds the transposed tile. K = 8192 rows:
        # 69 -> 31 us, 960 rows: 31 -> 10 us (mean over the projections of a decoder layer, rank 16 each).
        tiles = (N + 127) // 128
        rc = lib.axb_gemm_bf16(b.data_ptr(), b.stride(0), 1, a.data_ptr(), a.stride(0), 1, out.data_ptr(), out.stride(0), None, 0,
                               N, M, K, None, 0, None, 0, 0, float(alpha), 0.0, 6, min(max(1, _SM // tiles), (K + 63) // 64), 64,
                               _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
        _lib.check_rc(rc, "axb_gemm_bf16")
        return out
    if accumulate and splits <= 1 and out is not None and out.dtype == torch.float32 and c_in is None and a.is_cuda:
        # a single K pass owns every output tile: one sum per element (beta = 1) instead of split-K sums,
        # which also makes the launch eligible for the 2-CTA kernel
        return gemm(a, b, trans_a=trans_a, trans_b=trans_b, a2=a2, b2=b2, alpha=alpha, beta=1.0, c_in=out, out=out,
                    out_dtype=torch.float32, accumulate=False, splits=1, bn=bn)
    if accumulate:
        if out is None or out.dtype != torch.float32:
            raise ValueError("accumulate=True needs an fp32 `out`")
        out_mode = 2
    else:
        if splits > 1:
            raise ValueError("split-K needs accumulate=True (fp32 atomics)")
        out_mode = 0 if out_dtype == torch.bfloat16 else 1
        if out is None:
            out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    if out.stride(1) != 1:
        raise ValueError("gemm output must be row-major")
    if c_in is not None:
        if c_in.stride(1) != 1 or c_in.dtype != out.dtype:
            raise ValueError("c_in must be row-major with the output dtype")
    if glu is not None:
        _glu_launch(lib, glu, a, int(trans_a), b.data_ptr(), b.stride(0), int(trans_b), out, M, N, K, a2, b2, K2,
                    alpha, (None, 0, 0, 0, None, 0))
        return out
    if bn is None and _use_skinny(M, N, K, trans_a, trans_b, out, out_mode, c_in, beta):
        rows, cols = (M, N) if N <= 64 else (N, M)      # the long side is the kernel's 128-row operand
        p, s, p2, s2, mode = (a, b, a2, b2, 1) if N <= 64 else (b, a, b2, a2, 0)
        rc = lib.axb_gemm_skinny(
            p.data_ptr(), p.stride(0), s.data_ptr(), s.stride(0), out.data_ptr(), out.stride(0), rows, cols, K,
            _lib.ptr(p2), p2.stride(0) if p2 is not None else 0, _lib.ptr(s2), s2.stride(0) if s2 is not None else 0, K2,
            float(alpha), None, mode, out_mode, 0, 0.0, 1, 0, 0, _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
        _lib.check_rc(rc, "axb_gemm_skinny")
        return out
    pair = False
    if bn is None and accumulate:
        bn = _pick_bn(M, N)
    elif bn is None:
        epilogue = out_mode
        if c_in is not None and beta != 0.0:
            # what the kernels ask before they add by tile reductions (adds_by_tile)
            tiles = (out_mode == 1 and beta == 1.0 and c_in.data_ptr() == out.data_ptr() and c_in.stride(0) == out.stride(0)
                     and out.stride(0) % 4 == 0 and out.data_ptr() % 16 == 0)
            epilogue = 3 if tiles else 2
        bn, pair = _pick_tile(M, N, (K + 63) // 64 + (K2 + 63) // 64, epilogue)
    elif not accumulate:
        pair = _use_pair(M, N, bn)
    if pair:
        rc = lib.axb_gemm_bf16_pair(
            a.data_ptr(), a.stride(0), int(trans_a), b.data_ptr(), b.stride(0), int(trans_b),
            out.data_ptr(), out.stride(0), _lib.ptr(c_in), c_in.stride(0) if c_in is not None else 0, M, N, K,
            _lib.ptr(a2), a2.stride(0) if a2 is not None else 0, _lib.ptr(b2), b2.stride(0) if b2 is not None else 0,
            K2, float(alpha), float(beta if c_in is not None else 0.0), out_mode, None, 0, 0, 0, None, 0,
            _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
        _lib.check_rc(rc, "axb_gemm_bf16_pair")
        return out
    rc = lib.axb_gemm_bf16(
        a.data_ptr(), a.stride(0), int(trans_a),
        b.data_ptr(), b.stride(0), int(trans_b),
        out.data_ptr(), out.stride(0),
        _lib.ptr(c_in), c_in.stride(0) if c_in is not None else 0,
        M, N, K,
        _lib.ptr(a2), a2.stride(0) if a2 is not None else 0,
        _lib.ptr(b2), b2.stride(0) if b2 is not None else 0,
        K2, float(alpha), float(beta if c_in is not None else 0.0), out_mode, int(splits), int(bn),
        _lib.status_word(a.device).data_ptr(), _lib.stream_ptr(),
    )
    _lib.check_rc(rc, "axb_gemm_bf16")
    return out


def glu_fusable(M: int, I: int, device) -> bool:
    """Whether the GLU epilogues of the CTA-pair kernel serve an MLP with ``M`` token rows and ``I``
    intermediate columns (whole 32-column chunks; more than one 128-row tile, below that the short-side kernel is the
    faster one). They save a pass over gate|up whatever the number of tiles."""
    return USE_PAIR and USE_GLU_EPILOGUE and device.type == "cuda" and M > 128 and I % 32 == 0 and I >= 256


def _glu_launch(lib, glu, a, trans_a, b_ptr, ldb, trans_b, out, M, N, K, a2, b2, K2, alpha, pf):
    mode, kind, limit, other = glu
    if out is None or out.dtype != torch.bfloat16 or out.stride(1) != 1:
        raise ValueError("the GLU epilogue writes a row-major bf16 [M, 2I] `out`")
    if mode == "fwd":
        # b: [2I, K]; N passed by the caller is 2I
        I = N // 2
        h = other
        rc = lib.axb_gemm_bf16_pair_glu(
            a.data_ptr(), a.stride(0), trans_a, b_ptr, ldb, trans_b, out.data_ptr(), out.stride(0), None, 0,
            M, I, K, _lib.ptr(a2), a2.stride(0) if a2 is not None else 0, _lib.ptr(b2),
            b2.stride(0) if b2 is not None else 0, K2, float(alpha), 1, int(kind), float(limit or 0.0),
            h.data_ptr(), h.stride(0), *pf, _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
    else:
        gu = other
        rc = lib.axb_gemm_bf16_pair_glu(
            a.data_ptr(), a.stride(0), trans_a, b_ptr, ldb, trans_b, out.data_ptr(), out.stride(0),
            gu.data_ptr(), gu.stride(0), M, N, K, _lib.ptr(a2), a2.stride(0) if a2 is not None else 0,
            _lib.ptr(b2), b2.stride(0) if b2 is not None else 0, K2, float(alpha), 2, int(kind),
            float(limit or 0.0), None, 0, *pf, _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
    _lib.check_rc(rc, "axb_gemm_bf16_pair_glu")


def _use_skinny(M, N, K, trans_a, trans_b, out, out_mode, c_in, beta) -> bool:
    """The split-K cluster kernel of csrc/gemm_skinny.cu serves products with one side of a few columns, where 128-row tiles
    leave most SMs without a CTA. It gains what the split takes off the K loop and pays for the merge of the partial tiles, which
    grows with the short side: the lines are multiples of that side, by the CTAs that a tile gets (8 up to 33 tiles of the long
    side, 4 or 3 up to 92). Microseconds, ordinary tiles / this kernel, L2 flushed:

    N <= 64 (x A^T of an adapter). Up to 31 columns whatever the sizes: 192 x 4096 by 16 23.6 / 11.3, 8192 x 14336 by 16
    66.6 / 57.3, 65536 x 4096 by 16 109.6 / 104.4, 65536 x 512 by 16 level. Above: 1416 x 1496 by 56 19.3 / 15.3, 1576 x 608 by
    64 11.3 / 15.3; 8192 x 4096 by 48 29.7 / 27.7, 9216 x 2048 by 32 17.3 / 21.4, 9216 x 4096 by 64 27.9 / 33.7.
    M <= 128 (a generation step). Up to 16 rows, and 32 with a long K, whatever the weight: 16 x 4096 by 4096 1.35 times as fast,
    by 128256 1.10 times. Above: 64 x 14336 by 4096 1.54 times, 98 x 2000 by 624 17.4 / 15.3, 116 x 984 by 5192 15.3 / 19.4, 64 x
    2048 by 8192 0.89 times, 124 x 2608 by 18472 32.3 / 39.1, 128 x 4096 by 128256 0.92 times."""
    if trans_a or trans_b or out_mode > 1 or (c_in is not None and beta != 0.0) or K < 512 or out.stride(1) != 1:
        return False
    tiles = (max(M, N) + 127) // 128
    if N <= 64:
        return M > 128 and (N < 32 or (K >= 24 * N if tiles <= 33 else tiles <= 92 and K >= 80 * N))
    if M > 128 or N < 512:
        return False
    if M <= 16 or (M <= 32 and K >= 2048):
        return True
    pad = 32 if M <= 32 else 64 if M <= 64 else 128      # columns of the kernel's tile
    return K >= 20 * pad if tiles <= 33 else tiles <= 92 and K >= 40 * pad


def _use_pair(M, N, bn) -> bool:
    """Whether a tile width that the caller asked for means the CTA-pair kernel (256 x 256 tiles of an SM pair): from 74
    tiles on, one for every pair. Without a width ``_pick_tile`` decides, for fewer tiles too."""
    return USE_PAIR and bn == 256 and M >= 512 and N >= 512 and ((M + 255) // 256) * ((N + 255) // 256) >= 74


def _pick_bn(M, N) -> int:
    """Tile width of a split-K product (the split factor fills the SMs)."""
    m_tiles = (M + 127) // 128
    for bn in (256, 128, 64):
        if bn > 64 and N <= bn // 2:
            continue
        if m_tiles * ((N + bn - 1) // bn) >= _SM or bn == 64:
            return bn
    return 64


def pick_splits(out_tiles: int, k_blocks: int) -> int:
    """Split-K factor for skinny weight-gradient GEMMs so that all SMs get work."""
    if out_tiles >= _SM:
        return 1
    return max(1, min(k_blocks, _SM // max(out_tiles, 1)))


def _gemm_allgather(a, b_shard, info, *, trans_a, trans_b, a2, b2, alpha, beta, c_in, out, out_dtype, bn, glu=None):
    """GEMM against a row-sharded B. The full B is read from a staging buffer that an earlier
    launch filled; this launch's extra CTAs all-gather the next weight of the schedule (see
    parallel/fsdp.py)."""
    if trans_a:
        raise ValueError("the sharded-weight GEMM takes a row-major A")
    from ..parallel import symm as _symm  # noqa: F401  (registers the kernel signatures)

    lib = _lib.cuda_lib()
    a = _row_major_2d(a)
    M, Ka = a.shape
    rows, cols = info.rows, info.cols            # stored (full) B matrix
    N, K = (cols, rows) if trans_b else (rows, cols)
    if Ka != K:
        raise ValueError(f"gemm: inner dimensions differ ({Ka} vs {K})")
    K2 = 0
    if a2 is not None:
        a2, b2 = _row_major_2d(a2), _row_major_2d(b2)
        K2 = a2.shape[1]
    out_mode = 0 if out_dtype == torch.bfloat16 else 1
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype, device=a.device)
    bn, pair = _pick_tile(M, N, (K + 63) // 64 + (K2 + 63) // 64, out_mode) if bn is None else (bn, _use_pair(M, N, bn))
    ctx = info.ctx
    staging, plans = ctx.acquire(info, backward=trans_b)
    plan = None
    if plans and ctx.copy_engine:
        for pl in plans:          # copy engines: distance-1 and distance-2 weights, beside this GEMM
            ctx.prefetch_by_copy(pl)
            ctx.committed(pl)
        pf = (None, 0, 0, 0, None, 0)
    elif plans and plans[0][0].index in (info.index + 1, info.index - 1):
        plan = plans[0]           # gather CTAs of this launch: the next weight only
        nxt, slot = plan
        pf = (nxt.peer_bases_dev.data_ptr(), nxt.shard_offset, nxt.shard_bytes, nxt.world,
              ctx.staging[slot].data_ptr(), ctx.prefetch_ctas(nxt, 2.0 * M * N * K))
    else:
        pf = (None, 0, 0, 0, None, 0)
    if glu is not None:
        _glu_launch(lib, glu, a, 0, staging.data_ptr(), cols, int(trans_b), out, M, N, K, a2, b2, K2, alpha, pf)
    elif pair:
        rc = lib.axb_gemm_bf16_pair(
            a.data_ptr(), a.stride(0), 0, staging.data_ptr(), cols, int(trans_b), out.data_ptr(), out.stride(0),
            _lib.ptr(c_in), c_in.stride(0) if c_in is not None else 0, M, N, K,
            _lib.ptr(a2), a2.stride(0) if a2 is not None else 0, _lib.ptr(b2), b2.stride(0) if b2 is not None else 0,
            K2, float(alpha), float(beta if c_in is not None else 0.0), out_mode,
            *pf, _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
        _lib.check_rc(rc, "axb_gemm_bf16_pair")
    else:
        rc = lib.axb_gemm_bf16_prefetch(
            a.data_ptr(), a.stride(0), 0, staging.data_ptr(), cols, int(trans_b), out.data_ptr(), out.stride(0),
            _lib.ptr(c_in), c_in.stride(0) if c_in is not None else 0, M, N, K,
            _lib.ptr(a2), a2.stride(0) if a2 is not None else 0, _lib.ptr(b2), b2.stride(0) if b2 is not None else 0,
            K2, float(alpha), float(beta if c_in is not None else 0.0), out_mode, 1, int(bn),
            *pf, _lib.status_word(a.device).data_ptr(), _lib.stream_ptr())
        _lib.check_rc(rc, "axb_gemm_bf16_prefetch")
    if plan is not None:
        ctx.committed(plan)
    return out
