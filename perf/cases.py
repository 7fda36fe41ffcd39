"""What the framework is timed on: the work a training program has it do, through its public entry
points, from the smallest calls to the largest.

Every case is one pass a user's program makes again and again:
  block       `Sky1Block.forward` + `.backward` (dense or ragged batch, MHA or GQA)
  block_mx    `Sky1BlockMX.forward` + `.backward` (the block on MXFP8 products)
  lm          `Sky1LM.train_step` (embedding .. loss, backward, clipping, AdamW)
  linear      `ops.matmul` in the three forms a linear layer needs: forward, dgrad, and the weight
              gradient that accumulates into f32
  attention   `ops.attention_fwd` + `ops.attention_bwd` (dense or packed)
  rmsnorm     `ops.norm_fwd` with statistics + `ops.norm_bwd` with a residual gradient
  layernorm   `ops.norm_fwd` of the types and column counts outside the bf16 fast domain

The widths are the sky-1 model's own (hidden 2048, 16 heads of 128, FFN 5632, vocabulary 32768, and
narrower models of the same proportions); activations and output gradients are N(0, 1), weights
N(0, 0.02), norm gains near 1, tokens uniform.
"""
from __future__ import annotations

import math
import random

import torch

import cleanlm_b200 as cdl

HEAD_DIM = 128
VOCAB = 32768


def listed():
    return [
        # One short sequence at full width: the weights and the 28 launches are the whole cost.
        _block("block_1x256", batch=1, seq=256),
        # A ragged fine-tuning batch: six sequences of uneven length in 4003 rows, grouped-query heads.
        _block("block_ragged", batch=1, seq=4003, kv_heads=4, seqs=6, split=1),
        # The benchmark's training step: 8 sequences of 2048 tokens.
        _block("block_8x2048", batch=8, seq=2048),
        # The same step with block-scaled products.
        _block("block_mx_8x2048", kind="block_mx", batch=8, seq=2048),
        # A whole optimizer step of a shallow model with the real vocabulary: two microbatches.
        {"name": "lm_step", "kind": "lm", "layers": 2, "hidden": 2048, "batch": 2, "seq": 1024, "micro": 2},
        # A linear layer on few rows: operands are the weights, latency and launches count.
        _linear("linear_64", m=64, k=2048, n=5632),
        # A linear layer whose sizes leave every row off the 16-byte grid.
        _linear("linear_odd", m=1500, k=1027, n=2051),
        # A linear layer in f32 (a head or an adapter kept at full precision).
        _linear("linear_f32", m=1024, k=2048, n=1536, dtype="f32"),
        # Long-context attention, forward and backward.
        _attention("attention_8192", batch=1, seq=8192, heads=16, kv_heads=16),
        # Attention over a packed batch of short and middle-sized sequences with grouped-query heads.
        _attention("attention_packed", batch=1, seq=6144, heads=16, kv_heads=4, seqs=9, split=2),
        # The block's norm at the training shape, both directions.
        {"name": "rmsnorm_16384", "kind": "rmsnorm", "rows": 16384, "cols": 2048},
        # An f32 layer norm whose rows are not whole vectors of 8.
        {"name": "layernorm_f32", "kind": "layernorm", "rows": 8192, "cols": 2050, "x": "f32", "y": "f32"},
    ]


def _block(name, batch, seq, kind="block", hidden=2048, kv_heads=0, seqs=0, split=0):
    """kv_heads 0: as many as query heads; seqs 0: a dense batch, else that many ragged sequences."""
    return {"name": name, "kind": kind, "batch": batch, "seq": seq, "hidden": hidden, "kv_heads": kv_heads,
            "seqs": seqs, "split": split}


def _linear(name, m, k, n, dtype="bf16"):
    return {"name": name, "kind": "linear", "m": m, "k": k, "n": n, "dtype": dtype}


def _attention(name, batch, seq, heads, kv_heads, causal=True, seqs=0, split=0):
    return {"name": name, "kind": "attention", "batch": batch, "seq": seq, "heads": heads, "kv_heads": kv_heads,
            "causal": causal, "seqs": seqs, "split": split}


# --------------------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi, step=1):
    """An integer of [lo, hi], spread over the logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "block_mx", "lm", "linear", "linear", "linear_f32", "attention",
                       "attention", "rmsnorm", "layernorm"])
    if kind in ("block", "block_mx"):
        hidden = rng.choice([1024, 2048, 2048])
        mx = kind == "block_mx"
        tokens = _log_int(rng, 128, 16384, 128 if mx else 1)
        heads = hidden // HEAD_DIM
        kv = rng.choice([0, 0, heads // 4])
        seqs = 0 if mx else rng.choice([0, rng.randint(2, 9)])
        if seqs:  # few long sequences would cost more attention than the largest listed case
            return _pure(_block("", 1, min(max(tokens, 64 * seqs), 8192), kind, hidden, kv, seqs, rng.randrange(1000)))
        batch = rng.choice([b for b in (1, 2, 3, 4, 8) if tokens // b >= 128])
        seq = tokens // batch
        return _pure(_block("", batch, seq // 128 * 128 if mx else seq, kind, hidden, kv))
    if kind == "lm":
        return {"kind": "lm", "layers": rng.choice([1, 2]), "hidden": rng.choice([512, 1024, 2048]),
                "batch": rng.choice([1, 2]), "seq": _log_int(rng, 128, 1024), "micro": rng.choice([1, 2])}
    if kind == "linear":
        m, k, n = _log_int(rng, 16, 8192), _log_int(rng, 256, 6144), _log_int(rng, 256, 8192)
        if rng.random() < 0.6:  # layers of the usual widths; the rest is off the 16-byte grid
            k, n = (k + 63) // 64 * 64, (n + 63) // 64 * 64
        else:
            m, k, n = min(m, 2048), min(k, 2048) | 1, min(n, 4096) | 1
        return _pure(_linear("", m, k, n))
    if kind == "linear_f32":
        return _pure(_linear("", _log_int(rng, 16, 2048), _log_int(rng, 128, 2048), _log_int(rng, 128, 2048), "f32"))
    if kind == "attention":
        heads = rng.choice([8, 16])
        kv = rng.choice([heads, heads // 4])
        causal = rng.random() < 0.75
        if rng.random() < 0.5:
            seqs = rng.randint(2, 16)
            return _pure(_attention("", 1, _log_int(rng, 64 * seqs, 8192), heads, kv, causal, seqs, rng.randrange(1000)))
        batch = rng.choice([1, 2, 4])
        return _pure(_attention("", batch, _log_int(rng, 128, 8192 // batch), heads, kv, causal))
    rows = _log_int(rng, 64, 16384)
    if kind == "rmsnorm":
        return {"kind": "rmsnorm", "rows": rows, "cols": _log_int(rng, 256, 4096, 8)}
    return {"kind": "layernorm", "rows": rows, "cols": _log_int(rng, 100, 3000), "x": "f32",
            "y": rng.choice(["f32", "bf16"])}


def _pure(case):
    return {k: v for k, v in case.items() if k != "name"}


# --------------------------------------------------------------------------- inputs
def _lengths(case):
    """The sequence lengths of a ragged or packed case: uneven, at least 1, the last rows padding."""
    rng = random.Random(case["split"])
    total = case["seq"] - case["seq"] // 100  # up to one row in a hundred is padding
    w = [rng.uniform(0.2, 2.0) for _ in range(case["seqs"])]
    lens = [max(1, int(total * x / sum(w))) for x in w]
    lens[-1] += total - sum(lens)
    return lens


def _config(case):
    heads = case["hidden"] // HEAD_DIM
    return cdl.sky1.Sky1Config(batch=case["batch"], seqlen=case["seq"], hidden=case["hidden"], heads=heads,
                               kv_heads=case.get("kv_heads") or heads, head_dim=HEAD_DIM,
                               ffn=case["hidden"] * 11 // 4)


class _Random:
    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.gen, device="cuda") * std + mean).to(dtype)

    def tokens(self, *shape):
        return torch.randint(0, VOCAB, shape, generator=self.gen, device="cuda", dtype=torch.int32)


def _cumulative(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return torch.tensor(cu, dtype=torch.int32).cuda()


def _block_inputs(r, cfg):
    params = {n: r.normal(*shape, std=0.1, mean=1.0) if n.startswith("norm") else r.normal(*shape, std=0.02)
              for n, shape in cfg.param_shapes().items()}
    return params, r.normal(cfg.tokens, cfg.hidden), r.normal(cfg.tokens, cfg.hidden)


def prepare(case, seed):
    r = _Random(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("block", "block_mx"):
        cfg = _config(case)
        params, s["x"], s["dy"] = _block_inputs(r, cfg)
        if kind == "block_mx":
            s["block"] = cdl.sky1_mx.Sky1BlockMX(cfg, params)
        elif case["seqs"]:
            lens = _lengths(case)
            s["dy"][sum(lens):] = 0
            s["block"] = cdl.sky1.Sky1Block(cfg, params, cu_seqlens=_cumulative(lens), max_seqlen=max(lens))
        else:
            s["block"] = cdl.sky1.Sky1Block(cfg, params)
    elif kind == "lm":
        cfg = cdl.sky1.Sky1LMConfig(block=_config(case), layers=case["layers"], vocab=VOCAB, max_grad_norm=1.0)
        s["model"] = cdl.sky1.Sky1LM(cfg, seed=seed, init_on_device=True)
        s["tokens"] = r.tokens(case["micro"], cfg.block.tokens)
        s["targets"] = r.tokens(case["micro"], cfg.block.tokens)
    elif kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        dt = torch.float32 if case["dtype"] == "f32" else torch.bfloat16
        s["x"], s["w"], s["dy"] = r.normal(m, k, dtype=dt), r.normal(k, n, std=0.02, dtype=dt), r.normal(m, n, dtype=dt)
        s["gw"] = torch.zeros(k, n, device="cuda")
    elif kind == "attention":
        b, sq, h, hk = case["batch"], case["seq"], case["heads"], case["kv_heads"]
        lead = (sq,) if case["seqs"] else (b, sq)
        s["q"], s["k"], s["v"] = r.normal(*lead, h, HEAD_DIM), r.normal(*lead, hk, HEAD_DIM), r.normal(*lead, hk, HEAD_DIM)
        s["do"] = r.normal(*lead, h, HEAD_DIM)
        s["opts"] = cdl.ops.AttentionOpts(causal=case["causal"])
        if case["seqs"]:
            lens = _lengths(case)
            cu = _cumulative(lens)
            s["opts"] = cdl.ops.AttentionOpts(causal=case["causal"], cu_seqlens_q=cu, cu_seqlens_k=cu,
                                              max_seqlen_q=max(lens), max_seqlen_k=max(lens))
            s["rows"] = sum(lens)
    elif kind == "rmsnorm":
        rows, cols = case["rows"], case["cols"]
        s["x"], s["dy"], s["res"] = r.normal(rows, cols), r.normal(rows, cols), r.normal(rows, cols)
        s["scale"] = r.normal(cols, std=0.1, mean=1.0)
        s["dscale"] = torch.zeros(cols, device="cuda")
        s["opts"] = cdl.ops.NormFwdOpts(scale=s["scale"], save_stats=True)
    else:
        rows, cols = case["rows"], case["cols"]
        dt = {"f32": torch.float32, "bf16": torch.bfloat16}
        s["x"] = r.normal(rows, cols, dtype=dt[case["x"]])
        s["opts"] = cdl.ops.NormFwdOpts(scale=r.normal(cols, std=0.1, mean=1.0, dtype=torch.float32),
                                        bias=r.normal(cols, std=0.1, dtype=torch.float32), save_stats=True,
                                        norm_type="layer", out=dt[case["y"]])
    return s


# --------------------------------------------------------------------------- one pass
def run(s):
    kind = s["case"]["kind"]
    if kind in ("block", "block_mx"):
        out = s["block"].forward(s["x"])
        dx = s["block"].backward(s["dy"])
        return {"out": out, "dx": dx, "grads": s["block"].grads}
    if kind == "lm":
        model = s["model"]
        loss = model.train_step(s["tokens"], s["targets"])
        return {"loss": loss, "weights": model.master, "replica": model.replica, "m": model.m, "v": model.v}
    if kind == "linear":
        x, w, dy, gw = s["x"], s["w"], s["dy"], s["gw"]
        y = cdl.ops.matmul(x, w, cdl.ops.MatmulOpts(out=x.dtype))
        dx = cdl.ops.matmul(dy, w.T, cdl.ops.MatmulOpts(out=x.dtype))
        cdl.ops.matmul(x.T, dy, cdl.ops.MatmulOpts(out=torch.float32, c=gw, beta=1.0), out=gw)
        return {"y": y, "dx": dx, "gw": gw}
    if kind == "attention":
        q, k, v, do, opts = s["q"], s["k"], s["v"], s["do"], s["opts"]
        fwd = cdl.ops.attention_fwd(q, k, v, opts)
        dq, dk, dv = cdl.ops.attention_bwd(q, k, v, fwd.out, do, fwd.lse, opts)
        if opts.packed:  # rows after the last sequence are padding that no call writes
            n = s["rows"]
            return {"out": fwd.out[:n], "lse": fwd.lse[:, :n], "dq": dq[:n], "dk": dk[:n], "dv": dv[:n]}
        return {"out": fwd.out, "lse": fwd.lse, "dq": dq, "dk": dk, "dv": dv}
    if kind == "rmsnorm":
        f = cdl.ops.norm_fwd(s["x"], s["opts"])
        dx = cdl.ops.norm_bwd(s["x"], s["dy"], s["scale"], f.r_inv, s["dscale"], residual_dy=s["res"])
        return {"y": f.y, "r_inv": f.r_inv, "dx": dx, "dscale": s["dscale"]}
    f = cdl.ops.norm_fwd(s["x"], s["opts"])
    return {"y": f.y, "mean": f.mean, "r_inv": f.r_inv}


# --------------------------------------------------------------------------- what a pass cannot do without
def _attention_pairs(case):
    """(query, key) pairs that contribute, per head."""
    lens = _lengths(case) if case.get("seqs") else [case["seq"]] * case["batch"]
    return sum(n * (n + 1) / 2 if case.get("causal", True) else n * n for n in lens)


def _block_flops(case, cfg):
    hd = cfg.heads * cfg.head_dim
    per_token = 2.0 * (cfg.hidden * cfg.qkv_dim + hd * cfg.hidden + 3 * cfg.hidden * cfg.ffn)
    return 3 * per_token * cfg.tokens + 14.0 * hd * _attention_pairs(case)


def work(case):
    kind = case["kind"]
    if kind in ("block", "block_mx"):
        cfg = _config(case)
        params, act = cfg.param_count(), cfg.tokens * cfg.hidden
        # x, dy -> out, dx; weights read; f32 gradients read and written
        return {"bytes": 2.0 * (4 * act + params) + 8.0 * params, "flops": _block_flops(case, cfg)}
    if kind == "lm":
        cfg = _config(case)
        n = case["layers"] * cfg.param_count() + 2 * VOCAB * cfg.hidden + cfg.hidden
        head = 6.0 * cfg.tokens * cfg.hidden * VOCAB
        # master, both moments and the gradient buffer read and written, the bf16 replica written
        return {"bytes": 34.0 * n, "flops": case["micro"] * (case["layers"] * _block_flops(case, cfg) + head)}
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        e = 4 if case["dtype"] == "f32" else 2
        return {"bytes": e * (2.0 * m * k + k * n + 2.0 * m * n) + 8.0 * k * n, "flops": 6.0 * m * k * n}
    if kind == "attention":
        rows = case["batch"] * case["seq"] * HEAD_DIM
        # q, out, d_out, dq and k, v, dk, dv
        return {"bytes": 8.0 * rows * (case["heads"] + case["kv_heads"]),
                "flops": 14.0 * case["heads"] * HEAD_DIM * _attention_pairs(case)}
    n = float(case["rows"]) * case["cols"]
    if kind == "rmsnorm":
        return {"bytes": 10.0 * n + 8.0 * case["rows"], "flops": 16.0 * n}
    e = {"f32": 4, "bf16": 2}
    return {"bytes": (e[case["x"]] + e[case["y"]]) * n + 8.0 * case["rows"], "flops": 8.0 * n}


def tolerance(case):
    """About four times the relative error (2-norm) measured of the worst output of the kind:
    block       against f32 / f64 arithmetic on the same bf16 inputs: 3e-3 (out) .. 6.0e-3 (dWqkv)
    block_mx    another order of the attention's sums, one bf16 rounding carried through the E4M3
                roundings of the following products: 1e-2 (out) .. 3.5e-2 (dWqkv)
    lm          against f32 arithmetic: moments 1.1e-2 and 1.3e-2, weights 1.1e-3, loss 1.5e-5
    linear      against f64: bf16 results 1.7e-3; f32 operands 8.1e-7
    attention   against f64: 2.0e-3 (out) .. 2.5e-3 (dQ)
    rmsnorm     against f64: 1.7e-3, the rounding of bf16 results
    layernorm   against f64: f32 results 1.6e-7, bf16 results 1.7e-3
    """
    kind = case["kind"]
    if kind == "linear" and case["dtype"] == "f32":
        return {"rel": 4e-6}
    if kind == "layernorm" and case["y"] == "f32":
        return {"rel": 1e-6}
    return {"rel": {"block": 2.5e-2, "block_mx": 0.12, "lm": 5e-2, "linear": 7e-3, "attention": 1e-2, "rmsnorm": 7e-3,
                    "layernorm": 7e-3}[kind]}


# --------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """None: block_mx (its products are of quantized values) and lm (its state moves from pass to
    pass)."""
    kind = case["kind"]
    if kind in ("block_mx", "lm"):
        return None
    if kind == "block":
        return _exact_block(case, seed)
    s = prepare(case, seed)
    if kind == "linear":
        x, w, dy = s["x"].double(), s["w"].double(), s["dy"].double()
        return {"y": x @ w, "dx": dy @ w.T, "gw": x.T @ dy}
    if kind == "attention":
        return _exact_attention(case, s)
    x = s["x"].double()
    eps = s["opts"].eps
    if kind == "rmsnorm":
        dy, scale = s["dy"].double(), s["scale"].double()
        r = (x.square().mean(1) + eps).rsqrt()
        xh, g = x * r[:, None], dy * scale
        dx = r[:, None] * (g - xh * (g * xh).mean(1, keepdim=True)) + s["res"].double()
        return {"y": xh * scale, "r_inv": r, "dx": dx, "dscale": (dy * xh).sum(0)}
    mean = x.mean(1)
    r = ((x - mean[:, None]).square().mean(1) + eps).rsqrt()
    y = (x - mean[:, None]) * r[:, None] * s["opts"].scale.double() + s["opts"].bias.double()
    return {"y": y, "mean": mean, "r_inv": r}


def _spans(case):
    """(first row, rows) of every sequence, rows counted over the whole batch."""
    lens = _lengths(case) if case["seqs"] else [case["seq"]] * case["batch"]
    return [(sum(lens[:i]), n) for i, n in enumerate(lens)]


def _scores(q, k, causal):
    """q [n, heads, D], k [n, kv_heads, D] -> scaled (masked) scores [heads, n, n]."""
    k = k.repeat_interleave(q.shape[1] // k.shape[1], 1)
    sc = torch.einsum("qhd,khd->hqk", q, k) / math.sqrt(HEAD_DIM)
    if causal:
        sc = sc.masked_fill(torch.ones(sc.shape[1:], dtype=torch.bool, device=sc.device).triu(1), -math.inf)
    return sc


def _exact_attention(case, s):
    def rows(t):
        return t.reshape(-1, t.shape[-2], HEAD_DIM).double()

    q, k, v, do = (rows(s[n]) for n in ("q", "k", "v", "do"))
    out, dq, dk, dv = torch.zeros_like(q), torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    lse = torch.zeros(q.shape[1], q.shape[0], dtype=torch.float64, device="cuda")
    for first, n in _spans(case):
        r = slice(first, first + n)
        with torch.enable_grad():
            qi, ki, vi = (t[r].clone().requires_grad_() for t in (q, k, v))
            sc = _scores(qi, ki, case["causal"])
            o = torch.einsum("hqk,khd->qhd", sc.softmax(-1), vi.repeat_interleave(q.shape[1] // v.shape[1], 1))
            dq[r], dk[r], dv[r] = torch.autograd.grad(o, (qi, ki, vi), do[r])
        out[r], lse[:, r] = o.detach(), sc.detach().logsumexp(-1)
    if case["seqs"]:
        n = s["rows"]
        return {"out": out[:n], "lse": lse[:, :n], "dq": dq[:n], "dk": dk[:n], "dv": dv[:n]}
    lse = lse.reshape(-1, case["batch"], case["seq"]).transpose(0, 1)
    return {"out": out.reshape(s["q"].shape), "lse": lse, "dq": dq.reshape(s["q"].shape),
            "dk": dk.reshape(s["k"].shape), "dv": dv.reshape(s["v"].shape)}


def _exact_block(case, seed):
    cfg = _config(case)
    params, x, dy = _block_inputs(_Random(seed), cfg)
    spans = _spans(case)
    dy = dy.double()
    dy[sum(n for _, n in spans):] = 0
    w = {n: p.double().requires_grad_() for n, p in params.items()}
    x = x.double().requires_grad_()

    def norm(t, gain):
        return t * (t.square().mean(1, keepdim=True) + cfg.eps).rsqrt() * gain

    def rotated(t):
        angle = torch.outer(torch.arange(len(t), dtype=torch.float64, device="cuda"),
                            cfg.rope_base ** (-torch.arange(0, HEAD_DIM, 2, dtype=torch.float64, device="cuda") / HEAD_DIM))
        c, sn = angle.cos()[:, None], angle.sin()[:, None]
        lo, hi = t.chunk(2, -1)
        return torch.cat([lo * c - hi * sn, hi * c + lo * sn], -1)

    with torch.enable_grad():
        qkv = (norm(x, w["norm1"]) @ w["wqkv"]).view(cfg.tokens, -1, HEAD_DIM)
        parts = []
        for first, n in spans:
            q, k, v = qkv[first:first + n].split([cfg.heads, cfg.kv_heads, cfg.kv_heads], 1)
            p = _scores(rotated(q), rotated(k), True).softmax(-1)
            parts.append(torch.einsum("hqk,khd->qhd", p, v.repeat_interleave(cfg.heads // cfg.kv_heads, 1)))
        attn = torch.cat(parts).reshape(-1, cfg.heads * HEAD_DIM)
        attn = torch.nn.functional.pad(attn, (0, 0, 0, cfg.tokens - len(attn)))
        o = attn @ w["wo"] + x
        h = norm(o, w["norm2"])
        out = (torch.nn.functional.silu(h @ w["wgate"]) * (h @ w["wup"])) @ w["wdown"] + o
        grads = torch.autograd.grad(out, [x, *w.values()], dy)
    return {"out": out.detach(), "dx": grads[0], "grads": dict(zip(w, grads[1:]))}
