"""The work that users of this framework have it do most, as measurable cases.

Six kinds, each over the range of sizes that it meets:

* ``decode``: one generation step over a KV cache (chat, evaluation samples, GRPO rollouts), the loop body of
  ``models/kv_cache.py::generate_cached``; the batch is a multiple of 8 because that loop pads it;
* ``prefill``: the packed prompts of a batch through the model into a fresh part of the cache;
* ``train``: one whole optimizer step of the trainer on one packed row, LoRA adapters or every weight; rows are a
  multiple of 64 tokens because the collator pads them;
* ``attention``: packed variable-length attention, forward and backward, by head width and window;
* ``experts``: the routed experts of a sparse layer with NVFP4 weights and expert adapters, forward and backward;
* ``head``: the loss of a frozen output projection over a large vocabulary, forward and backward.

Models are cut to a few layers of the named width: every layer of a full model repeats the same work."""
import math

import numpy as np
import torch

from axolotl_b200.models.config import ModelConfig
from axolotl_b200.models.kv_cache import KVCache, _DecodeMeta, _PrefillMeta
from axolotl_b200.models.lora import ALL_LINEAR, LoraSpec, inject_lora
from axolotl_b200.models.moe import Experts
from axolotl_b200.models.transformer import CausalLM
from axolotl_b200.ops import functional as Fn
from axolotl_b200.ops.grouped import bump_param_epoch, moe_local_forward
from axolotl_b200.ops.lora import linear
from axolotl_b200.ops.nvfp4 import quantize_nvfp4
from axolotl_b200.train.optimizer import FlatAdamW, build_param_groups, make_lr_lambda
from axolotl_b200.train.trainer import TrainArgs, Trainer

DEV = "cuda"
EPS, THETA = 1e-5, 500000.0
LORA_R, LORA_ALPHA = 16, 32

# (hidden, intermediate, query heads, key / value heads, head width, vocabulary): the headline 8B model, an 8B model
# with a narrower MLP, and a small model
WIDTHS = {"8b": (4096, 14336, 32, 8, 128, 128256), "8b_narrow": (4096, 12288, 32, 8, 128, 151936),
          "1b": (2048, 5632, 32, 4, 64, 32000)}


def listed():
    return [
        # the smallest call: one chat user on a small model, a few hundred tokens into the conversation
        dict(name="decode_small_model", kind="decode", width="1b", layers=8, batch=8, shortest=60, longest=300),
        # one chat user on the 8B model
        dict(name="decode_chat_8b", kind="decode", width="8b", layers=4, batch=8, shortest=200, longest=900),
        # a rollout batch of reinforcement learning, deep into its completions
        dict(name="decode_rollout_8b", kind="decode", width="8b", layers=4, batch=64, shortest=500, longest=4096),
        # the prompts of such a batch, of odd lengths
        dict(name="prefill_8b", kind="prefill", width="8b", layers=4, batch=13, tokens=4777),
        # a short fine-tuning row: a few chat samples, micro-batch 1
        dict(name="lora_short_row_8b", kind="train", width="8b", layers=2, tokens=960, shortest=64, longest=500, lora=True),
        # the headline row: samples of 256 to 4096 tokens packed to 8192
        dict(name="lora_packed_row_8b", kind="train", width="8b", layers=2, tokens=8192, shortest=256, longest=4096, lora=True),
        # full fine-tuning of a small model
        dict(name="full_tune_1b", kind="train", width="1b", layers=4, tokens=4096, shortest=100, longest=2048, lora=False),
        # one long document (context extension)
        dict(name="attention_long", kind="attention", hq=32, hk=8, d=128, tokens=16384, docs=1, window=0),
        # many short samples in one row, sliding-window layers with 64-wide heads
        dict(name="attention_window_d64", kind="attention", hq=64, hk=8, d=64, tokens=7777, docs=11, window=128),
        # 256-wide heads
        dict(name="attention_wide_d256", kind="attention", hq=16, hk=8, d=256, tokens=8192, docs=4, window=0),
        # a training micro-batch through 128 experts
        dict(name="experts_8k", kind="experts", tokens=8192, experts=128, topk=8, hidden=2048, inter=768),
        # a short one: most experts see a few rows
        dict(name="experts_short", kind="experts", tokens=333, experts=128, topk=8, hidden=2048, inter=768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "train", "attention", "experts", "head"])
    if kind == "decode":
        width = rng.choice(sorted(WIDTHS))
        longest = _log(rng, 32, 4096)
        return dict(kind=kind, width=width, layers=rng.randint(2, 4), batch=8 * _log(rng, 1, 8),
                    shortest=max(1, int(longest * rng.random())), longest=longest)
    if kind == "prefill":
        tokens = _log(rng, 20, 6000)
        return dict(kind=kind, width=rng.choice(sorted(WIDTHS)), layers=rng.randint(2, 4), batch=_log(rng, 1, min(64, tokens // 10)), tokens=tokens)
    if kind == "train":
        lora = rng.random() < 0.7
        tokens = 64 * _log(rng, 4, 96 if lora else 64)
        longest = max(16, int(tokens * rng.uniform(0.1, 1.0)))
        return dict(kind=kind, width=rng.choice(sorted(WIDTHS)) if lora else "1b", layers=rng.randint(1, 2), tokens=tokens,
                    shortest=max(4, longest // 8), longest=longest, lora=lora)
    if kind == "attention":
        d = rng.choice([64, 128, 128, 256])
        hk = rng.choice([2, 4, 8])
        tokens = _log(rng, 200, 12000)
        return dict(kind=kind, hq=hk * rng.choice([1, 2, 4]), hk=hk, d=d, tokens=tokens, docs=_log(rng, 1, max(1, min(40, tokens // 40))),
                    window=rng.choice([0, 0, _log(rng, 64, 4096)]) if d != 256 else 0)
    if kind == "experts":
        return dict(kind=kind, tokens=_log(rng, 100, 8192), experts=rng.choice([32, 64, 128]), topk=rng.choice([2, 4, 8]),
                    hidden=rng.choice([1024, 2048]), inter=rng.choice([512, 768, 1024]))
    return dict(kind=kind, tokens=64 * _log(rng, 4, 96), hidden=256 * rng.randint(4, 16), vocab=8 * _log(rng, 4000, 19000))


# ------------------------------------------------------------------------------------------------ inputs
def _lengths(r, count, lo, hi):
    return [int(v) for v in r.integers(lo, hi + 1, size=count)]


def _packed(r, total, lo, hi):
    """Document lengths that fill ``total`` tokens."""
    out, left = [], total
    while left > 0:
        n = min(left, int(r.integers(lo, hi + 1)))
        out.append(n)
        left -= n
    return out


def _documents(r, total, docs):
    """``docs`` lengths of one token or more that sum to ``total``."""
    cuts = np.sort(r.choice(np.arange(1, total), size=docs - 1, replace=False)) if docs > 1 else np.array([], dtype=np.int64)
    return np.diff(np.concatenate([[0], cuts, [total]])).astype(int).tolist()


def _model(case, seed):
    H, I, hq, hk, d, V = WIDTHS[case["width"]]
    cfg = ModelConfig(model_type="llama", vocab_size=V, hidden_size=H, intermediate_size=I, num_hidden_layers=case["layers"],
                      num_attention_heads=hq, num_key_value_heads=hk, head_dim=d, rms_norm_eps=EPS, rope_theta=THETA,
                      max_position_embeddings=8192)
    torch.manual_seed(seed)
    return CausalLM(cfg, dtype=torch.bfloat16, device=DEV).init_weights(seed)


def _cover(f):
    """Ones in the diagonal blocks of a fused projection's B: each sub-projection has an adapter of its own."""
    out = torch.zeros_like(f.lora_B)
    for r0, rows, c0, cols in f.lora_blocks:
        out[r0:r0 + rows, c0:c0 + cols] = 1.0
    return out


def prepare(case, seed):
    r = np.random.default_rng(seed)
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    if kind == "decode":
        m = _model(case, seed).eval()
        lens = _lengths(r, case["batch"], case["shortest"], case["longest"])
        cache = KVCache(m, case["batch"], case["longest"] + 64)
        for t in (cache.k, cache.v):
            t.normal_(0.0, 1.0, generator=g)
        token = torch.randint(0, m.config.vocab_size, (case["batch"],), device=DEV, generator=g)
        return dict(case=case, model=m, cache=cache, token=token, pos=torch.tensor(lens, dtype=torch.long, device=DEV),
                    seq=torch.arange(case["batch"], device=DEV))
    if kind == "prefill":
        m = _model(case, seed).eval()
        lens = _documents(r, case["tokens"], case["batch"])
        pad = (-sum(lens)) % 8
        cache = KVCache(m, case["batch"], max(lens) + 64)
        cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
        seq = [b for b, n in enumerate(lens) for _ in range(n)] + [0] * pad
        pos = [i for n in lens for i in range(n)]
        t = lambda v, k=torch.long: torch.tensor(v, dtype=k, device=DEV)  # noqa: E731
        ids = torch.randint(0, m.config.vocab_size, (sum(lens) + pad,), device=DEV, generator=g)
        return dict(case=case, model=m, cache=cache, cu=list(cu) + ([int(cu[-1]) + pad] if pad else []), ids=ids[None], lens=lens,
                    pos=t(pos + list(range(pad)), torch.int32)[None], seq=t(seq), slot=t(pos + [cache.max_len - 1] * pad),
                    last=t([int(c) - 1 for c in cu[1:]]))
    if kind == "train":
        m = _model(case, seed)
        if case["lora"]:
            inject_lora(m, LoraSpec(r=LORA_R, lora_alpha=LORA_ALPHA, target_modules=list(ALL_LINEAR)))
            with torch.no_grad():      # adapters as a run in progress has them (B is zero only in the very first step)
                for n, p in m.named_parameters():
                    if "lora_" in n:
                        p.normal_(0.0, 0.02, generator=g)
                        p.copy_(p.bfloat16())
                for _, f in m.fused_linears():
                    f.lora_B.mul_(_cover(f))
            m.refresh_lora_shadows()
        opt = FlatAdamW(build_param_groups(m.named_parameters(), weight_decay=0.0), lr=1e-4, max_grad_norm=1.0)
        opt.bind_model_shadows(m)
        tr = Trainer(m, opt, make_lr_lambda("constant", 10 ** 9, 0), TrainArgs(max_steps=10 ** 9, learning_rate=1e-4, include_tkps=False),
                     lambda e: [], device=torch.device(DEV))
        m.train()
        T = case["tokens"]
        lens = _packed(r, T, case["shortest"], case["longest"])
        ids = torch.from_numpy(r.integers(3, m.config.vocab_size, size=(1, T)))
        labels = ids.clone()
        at = 0
        for n in lens:                 # the prompt's share of every sample is not trained on
            labels[0, at:at + max(1, n // 5)] = -100
            at += n
        pos = torch.from_numpy(np.concatenate([np.arange(n) for n in lens]).astype(np.int64))[None]
        batch = dict(input_ids=ids.pin_memory(), labels=labels.pin_memory(), position_ids=pos.pin_memory())
        state = {}
        for grp in opt.groups:
            for n, p, o, k in grp["entries"]:
                state[n] = (grp["master"][o:o + k].view(p.shape), grp["exp_avg"][o:o + k].view(p.shape))
        return dict(case=case, model=m, opt=opt, trainer=tr, batch=batch, lens=lens, state=state)
    if kind == "attention":
        hq, hk, d, T = case["hq"], case["hk"], case["d"], case["tokens"]
        lens = _documents(r, T, case["docs"])
        meta = Fn.AttnMeta(np.concatenate([[0], np.cumsum(lens)]), torch.device(DEV))
        qkv = torch.empty(T, (hq + 2 * hk) * d, dtype=torch.bfloat16, device=DEV).normal_(0.0, 1.0, generator=g)
        dout = torch.empty(T, hq * d, dtype=torch.bfloat16, device=DEV).normal_(0.0, 1.0, generator=g)
        return dict(case=case, meta=meta.windowed(case["window"]) if case["window"] else meta, lens=lens, qkv=qkv.requires_grad_(True), dout=dout)
    if kind == "experts":
        T, E, k, H, I = case["tokens"], case["experts"], case["topk"], case["hidden"], case["inter"]
        torch.manual_seed(seed)
        ex = Experts(E, H, I, "silu", torch.bfloat16, DEV)
        q = {}
        for which, shape in (("gate_up", (E, 2 * I, H)), ("down", (E, H, I))):
            qd, sc, pts = quantize_nvfp4(torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(0.0, 0.02, generator=g))
            q[which] = {"qdata": qd, "scale": sc, "pts": pts.reshape(-1)}
        ex.nvfp4, ex.gate_up_proj, ex.down_proj = q, None, None
        ex.add_lora(LORA_R, LORA_ALPHA)
        with torch.no_grad():
            for p in ex.lora.values():
                p.normal_(0.0, 0.02, generator=g)
                p.copy_(p.bfloat16())
        x = torch.empty(T, H, dtype=torch.bfloat16, device=DEV).normal_(0.0, 1.0, generator=g).requires_grad_(True)
        # a router with some experts more popular than others
        score = torch.empty(T, E, device=DEV).normal_(0.0, 1.0, generator=g) + 0.5 * torch.empty(E, device=DEV).normal_(0.0, 1.0, generator=g)
        w, idx = torch.topk(torch.softmax(score, -1), k, -1)
        dy = torch.empty(T, H, dtype=torch.bfloat16, device=DEV).normal_(0.0, 1.0, generator=g)
        return dict(case=case, experts=ex, x=x, w=(w / w.sum(-1, keepdim=True)).requires_grad_(True), idx=idx, dy=dy)
    T, H, V = case["tokens"], case["hidden"], case["vocab"]
    h = torch.empty(T, H, dtype=torch.bfloat16, device=DEV).normal_(0.0, 1.0, generator=g).requires_grad_(True)
    W = torch.empty(V, H, dtype=torch.bfloat16, device=DEV).normal_(0.0, 0.02, generator=g)
    labels = torch.randint(0, V, (T,), device=DEV, generator=g)
    labels[torch.rand(T, device=DEV, generator=g) < 0.2] = -100
    return dict(case=case, h=h, W=W, labels=labels, items=int((labels != -100).sum()))


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "decode":
        with torch.no_grad():
            m, pos = s["model"], s["pos"]
            meta = _DecodeMeta(s["cache"], s["seq"], pos, True)
            out = m(s["token"][None], pos.to(torch.int32)[None], attn_meta=meta, return_logits=False)
            logits = linear(out.hidden_states.reshape(pos.numel(), -1), m.output_weight()).float()
        return dict(logits=logits, k=s["cache"].k, v=s["cache"].v)
    if kind == "prefill":
        with torch.no_grad():
            m = s["model"]
            meta = _PrefillMeta(s["cache"], Fn.AttnMeta(s["cu"], torch.device(DEV)), s["seq"], s["slot"])
            out = m(s["ids"], s["pos"], attn_meta=meta, return_logits=False)
            h = out.hidden_states.reshape(-1, out.hidden_states.shape[-1])
            logits = linear(h[s["last"]], m.output_weight()).float()
        n = sum(s["lens"])
        return dict(logits=logits, hidden=h[:n])
    if kind == "train":
        loss = s["trainer"].training_step([s["batch"]])
        return dict(loss=loss, **{n: list(v) for n, v in s["state"].items()})
    if kind == "attention":
        c = s["case"]
        out = Fn.flash_varlen(s["qkv"], s["meta"], c["hq"], c["hk"], c["d"])
        return dict(out=out.detach(), dqkv=torch.autograd.grad(out, s["qkv"], s["dout"])[0])
    if kind == "experts":
        ex = s["experts"]
        y = moe_local_forward(ex, s["x"], s["w"], s["idx"], s["case"]["experts"])
        names = sorted(ex.lora.keys())
        grads = torch.autograd.grad(y, [s["x"], s["w"]] + [ex.lora[n] for n in names], s["dy"])
        bump_param_epoch()             # as the trainer does after its step: adapters are about to change
        return dict(y=y.detach(), **dict(zip(["dx", "dw"] + names, grads)))
    loss = Fn.linear_cross_entropy(s["h"], s["W"], s["labels"], num_items=s["items"])
    return dict(loss=loss.detach(), dh=torch.autograd.grad(loss, s["h"])[0])


# ------------------------------------------------------------------------------------------------ what it cannot do without
def _pairs(lens, window=0):
    """Query-key pairs of causal attention."""
    return float(sum(n * (n + 1) / 2 if not window or n <= window else window * (window + 1) / 2 + (n - window) * window for n in lens))


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prefill", "train"):
        H, I, hq, hk, d, V = WIDTHS[case["width"]]
        L = case["layers"]
        layer = H * (hq + 2 * hk) * d + hq * d * H + 3 * H * I
        mean = (case["shortest"] + case["longest"]) / 2 if kind != "prefill" else 2 * case["tokens"] / (case["batch"] + 1)
    if kind == "decode":
        B = case["batch"]
        kv = L * B * mean * 2 * hk * d
        return {"bytes": 2 * (L * layer + V * H) + 2 * kv + 4 * B * V, "flops": 2 * B * (L * layer + V * H) + 4 * L * B * mean * hq * d}
    if kind == "prefill":
        B, T = case["batch"], case["tokens"]
        return {"bytes": 2 * (L * layer + V * H) + T * 2 * H + 4 * T * L * hk * d + 4 * B * V,
                "flops": 2 * T * L * layer + 2 * B * V * H + 4 * L * hq * d * T * mean / 2}
    if kind == "train":
        T = case["tokens"]
        times = 4 if case["lora"] else 6           # forward and input gradient, and the weight gradient where weights train
        adapters = L * LORA_R * (3 * H + (hq + 2 * hk) * d + hq * d + H + 2 * H + 2 * I + I + H)
        trained = adapters if case["lora"] else L * (layer + 2 * H) + H + 2 * V * H
        att = L * 4 * hq * d * 3.5 * T * mean / 2
        states = 4 * trained * 6 + 2 * trained     # master and moments read and written, bf16 copy written
        act = L * T * 2 * (4 * H + 2 * (hq + 2 * hk) * d + 4 * I) * 2
        # a frozen layer's input gradient below the first adapter is part of the step; the embedding gradient is a scatter
        flops = times * T * L * layer + times * T * V * H + att + (6 * T * adapters if case["lora"] else 0)
        return {"bytes": 2 * 2 * (L * layer + V * H) + states + act, "flops": flops}
    if kind == "attention":
        hq, hk, d, T = case["hq"], case["hk"], case["d"], case["tokens"]
        n = T / case["docs"]
        pairs = case["docs"] * _pairs([n], case["window"])
        if case["docs"] > 1 and not case["window"]:
            pairs *= 2 * case["docs"] / (case["docs"] + 1)       # mean square of uniformly cut lengths
        return {"bytes": 2 * T * d * (4 * (hq + 2 * hk) + 0) * 0.75 + 2 * T * d * hq * 3, "flops": 14.0 * hq * d * pairs}
    if kind == "experts":
        T, E, k, H, I = case["tokens"], case["experts"], case["topk"], case["hidden"], case["inter"]
        used = E * (1 - (1 - k / E) ** T)
        S, W = T * k, 3 * H * I
        r = LORA_R
        return {"bytes": 2 * used * W * (0.5 + 1 / 16) + 2 * T * H * 5 + 4 * 3 * E * r * (H + 2 * I + I + H) + 2 * S * (3 * I),
                "flops": 4.0 * S * W + 8.0 * S * r * (2 * H + 3 * I)}
    T, H, V = case["tokens"], case["hidden"], case["vocab"]
    return {"bytes": 2 * 2 * V * H + 2 * T * H * 2, "flops": 4.0 * T * H * V}


# What bf16 operands and bf16 intermediate results give (measured against `exact`, about four times what was seen; the
# difference of two such implementations is at most of that size).
_TOL = {"decode": 0.03, "prefill": 0.03, "train": 0.03, "attention": 0.012, "experts": 0.02, "head": 0.015}


def tolerance(case):
    return {"rel": _TOL[case["kind"]], "max": 0.99 if case["kind"] == "train" else 0.5}


# ------------------------------------------------------------------------------------------------ 64-bit results
class _Attention64(torch.autograd.Function):
    """Causal (windowed) attention of every document in 64 bits, one key / value head and one block of queries at a time."""

    @staticmethod
    def _blocks(lens, window):
        at = 0
        for n in lens:
            for q0 in range(0, n, 2048):
                q1 = min(n, q0 + 2048)
                k0 = max(0, q0 - window + 1) if window else 0
                qi, ki = torch.arange(q0, q1, device=DEV)[:, None], torch.arange(k0, q1, device=DEV)[None]
                off = (ki > qi) | ((ki <= qi - window) if window else False)
                yield at + q0, at + q1, at + k0, at + q1, off
            at += n

    @staticmethod
    def forward(ctx, q, k, v, lens, window):
        T, hq, d = q.shape
        hk = k.shape[1]
        G = hq // hk
        out = torch.empty_like(q)
        for a, b, c, e, off in _Attention64._blocks(lens, window):
            for h in range(hk):
                s = q[a:b, h * G:(h + 1) * G].transpose(0, 1) @ k[c:e, h].t() / math.sqrt(d)
                out[a:b, h * G:(h + 1) * G] = (s.masked_fill_(off, -math.inf).softmax(-1) @ v[c:e, h]).transpose(0, 1)
        ctx.save_for_backward(q, k, v)
        ctx.args = lens, window
        return out

    @staticmethod
    def backward(ctx, do):
        q, k, v = ctx.saved_tensors
        lens, window = ctx.args
        T, hq, d = q.shape
        hk = k.shape[1]
        G = hq // hk
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for a, b, c, e, off in _Attention64._blocks(lens, window):
            for h in range(hk):
                qq, dd = (t[a:b, h * G:(h + 1) * G].transpose(0, 1) for t in (q, do))
                p = (qq @ k[c:e, h].t() / math.sqrt(d)).masked_fill_(off, -math.inf).softmax(-1)
                dp = dd @ v[c:e, h].t()
                ds = p * (dp - (p * dp).sum(-1, keepdim=True)) / math.sqrt(d)
                dq[a:b, h * G:(h + 1) * G] = (ds @ k[c:e, h]).transpose(0, 1)
                dk[c:e, h] += torch.einsum("gqk,gqd->kd", ds, qq)
                dv[c:e, h] += torch.einsum("gqk,gqd->kd", p, dd)
        return dq, dk, dv, None, None


def _rms64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _rope64(x, pos):
    d = x.shape[-1]
    inv = 1.0 / (THETA ** (torch.arange(0, d, 2, dtype=torch.float64, device=DEV) / d))
    a = pos.double()[:, None, None] * inv
    c, s = a.cos(), a.sin()
    x1, x2 = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)


class _Linear64(torch.autograd.Function):
    """x W^T for a frozen 16-bit W, widened a part at a time."""

    @staticmethod
    def forward(ctx, x, W):
        ctx.W = W
        return torch.cat([x @ w.double().t() for w in W.split(16384)], -1)

    @staticmethod
    def backward(ctx, dy):
        return sum(d @ w.double() for d, w in zip(dy.split(16384, -1), ctx.W.split(16384))), None


def _layers64(case, h, pos, par, attend):
    """The decoder layers; ``par(name, x)`` applies the named projection, ``par(name)`` is the named norm weight."""
    H, I, hq, hk, d, V = WIDTHS[case["width"]]
    for i in range(case["layers"]):
        p = "layers.%d." % i
        x = _rms64(h, par(p + "input_layernorm"))
        q, k, v = par(p + "self_attn.qkv_proj", x).split([hq * d, hk * d, hk * d], -1)
        q, k = _rope64(q.reshape(-1, hq, d), pos), _rope64(k.reshape(-1, hk, d), pos)
        a = attend(i, q, k, v.reshape(-1, hk, d))
        h = h + par(p + "self_attn.o_proj", a.reshape(-1, hq * d))
        g, u = par(p + "mlp.gate_up_proj", _rms64(h, par(p + "post_attention_layernorm"))).chunk(2, -1)
        h = h + par(p + "mlp.down_proj", torch.nn.functional.silu(g) * u)
    return _rms64(h, par("norm"))


def _loss64(h, W, labels, items):
    """Cross entropy of h W^T, a few rows at a time; its gradient with respect to h (and W, where it trains)."""
    loss, dh, dW = 0.0, torch.zeros_like(h), torch.zeros(W.shape, dtype=torch.float64, device=DEV) if W.dtype == torch.float64 else None
    for a in range(0, h.shape[0], 1024):
        hh = h[a:a + 1024].detach()
        z = _Linear64.apply(hh, W)
        lab = labels[a:a + 1024]
        on = lab != -100
        lse = torch.logsumexp(z, -1)
        loss += float((lse - z.gather(1, lab.clamp(min=0)[:, None])[:, 0])[on].sum())
        z = (z - lse[:, None]).exp_()
        z[torch.arange(len(lab), device=DEV), lab.clamp(min=0)] -= 1.0
        z *= on[:, None] / items
        dh[a:a + 1024] = sum(d @ w.double() for d, w in zip(z.split(16384, -1), W.split(16384)))
        if dW is not None:
            dW += z.t() @ hh
    return loss / items, dh, dW


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        m = s["model"]
        P = dict(m.named_parameters())
        with torch.no_grad():
            par = lambda n, x=None: P[n + ".weight"].double() if x is None else _Linear64.apply(x, P[n + ".weight"])  # noqa: E731
            if kind == "decode":
                pos, B = s["pos"], case["batch"]
                ck, cv = s["cache"].k.double(), s["cache"].v.double()

                def attend(i, q, k, v):
                    out = torch.empty_like(q)
                    for b in range(B):
                        n = int(pos[b])
                        ck[i, b, n], cv[i, b, n] = k[b].reshape(-1), v[b].reshape(-1)
                        kk, vv = (t[i, b, :n + 1].view(n + 1, k.shape[1], -1).transpose(0, 1) for t in (ck, cv))
                        qq = q[b].view(k.shape[1], -1, q.shape[-1])
                        out[b] = ((qq @ kk.transpose(1, 2) / math.sqrt(q.shape[-1])).softmax(-1) @ vv).reshape(q.shape[1], -1)
                    return out

                h = _layers64(case, m.embed_tokens[s["token"]].double(), pos, par, attend)
                return dict(logits=_Linear64.apply(h, m.output_weight()), k=ck, v=cv)
            n = sum(s["lens"])
            h = _layers64(case, m.embed_tokens[s["ids"][0, :n]].double(), s["pos"][0, :n], par,
                          lambda i, q, k, v: _Attention64.apply(q, k, v, s["lens"], 0))
            return dict(logits=_Linear64.apply(h[s["last"]], m.output_weight()), hidden=h)
    if kind == "train":
        m, lr = s["model"], 1e-4
        P = dict(m.named_parameters())
        leaf = {n: P[n].detach().double().requires_grad_(True) for n in s["state"]}
        of = lambda n: leaf[n] if n in leaf else P[n].detach().double()  # noqa: E731

        def par(n, x=None):
            if x is None:
                return of(n + ".weight")
            if not case["lora"]:
                return x @ of(n + ".weight").t()
            mod = m.get_submodule(n)
            low = (LORA_ALPHA / LORA_R) * (x @ leaf[n + ".lora_A"].t())
            return _Linear64.apply(x, P[n + ".weight"].detach()) + low @ (leaf[n + ".lora_B"] * _cover(mod)).t()

        ids, lab = s["batch"]["input_ids"][0].to(DEV), s["batch"]["labels"][0].to(DEV)
        lab = torch.cat([lab[1:], lab.new_full((1,), -100)])
        h = _layers64(case, of("embed_tokens")[ids], s["batch"]["position_ids"][0].to(DEV), par,
                      lambda i, q, k, v: _Attention64.apply(q, k, v, s["lens"], 0))
        W = of("lm_head") if "lm_head" in leaf else P["lm_head"].detach()
        loss, dh, dW = _loss64(h, W.detach(), lab, int((lab != -100).sum()))
        h.backward(dh)
        if dW is not None:
            leaf["lm_head"].grad = dW
        norm = math.sqrt(sum(float(t.grad.pow(2).sum()) for t in leaf.values()))
        clip, out = min(1.0, 1.0 / (norm + 1e-6)), {}
        for n, t in leaf.items():
            gr = t.grad * clip
            out[n] = [t.detach() - lr * gr / (gr.abs() + 1e-8), 0.1 * gr]
        return dict(loss=torch.tensor(loss, dtype=torch.float64), **out)
    if kind == "attention":
        hq, hk, d, T = case["hq"], case["hk"], case["d"], case["tokens"]
        x = s["qkv"].detach().double()
        q, k, v = (t.reshape(T, -1, d).contiguous().requires_grad_(True) for t in x.split([hq * d, hk * d, hk * d], -1))
        out = _Attention64.apply(q, k, v, s["lens"], case["window"])
        out.backward(s["dout"].double().view(T, hq, d))
        return dict(out=out.detach().reshape(T, -1), dqkv=torch.cat([t.grad.reshape(T, -1) for t in (q, k, v)], -1))
    if kind == "experts":
        ex, E, k, H = s["experts"], case["experts"], case["topk"], case["hidden"]
        grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device=DEV)
        grid = torch.cat([grid, -grid])

        def weight(which, e):
            q = ex.nvfp4[which]
            b = q["qdata"][e].long()
            val = torch.stack([grid[b & 15], grid[b >> 4]], -1).reshape(b.shape[0], -1)
            return val * q["scale"][e].float().double().repeat_interleave(16, -1) * q["pts"][e].double()

        x = s["x"].detach().double().requires_grad_(True)
        w = s["w"].detach().double().requires_grad_(True)
        lo = {n: p.detach().double().requires_grad_(True) for n, p in ex.lora.items()}
        sc = LORA_ALPHA / LORA_R

        def proj(v, which, e):
            A = lo[which + "_A"][e * LORA_R:(e + 1) * LORA_R]
            B = lo[which + "_B"].view(-1, LORA_R, E)[:, :, e]
            return v @ weight(which, e).t() + sc * (v @ A.t()) @ B.t()

        y = torch.zeros(s["x"].shape, dtype=torch.float64, device=DEV)
        for e in range(E):
            tok, slot = (s["idx"] == e).nonzero(as_tuple=True)
            if len(tok):
                gt, up = proj(x[tok], "gate_up", e).chunk(2, -1)
                part = proj(torch.nn.functional.silu(gt) * up, "down", e) * w[tok, slot][:, None]
                part.backward(s["dy"].double()[tok])      # each expert's graph on its own: weights are widened one at a time
                y.index_add_(0, tok, part.detach())
        zero = lambda t: t.grad if t.grad is not None else torch.zeros_like(t)  # noqa: E731
        return dict(y=y, dx=zero(x), dw=zero(w), **{n: zero(p) for n, p in lo.items()})
    loss, dh, _ = _loss64(s["h"].detach().double(), s["W"], s["labels"], s["items"])
    return dict(loss=torch.tensor(loss, dtype=torch.float64), dh=dh)
