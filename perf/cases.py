"""Performance cases: the work that training and evaluating a hybrid mixture-of-experts model puts on this
framework, through its public entry points.

A case is a dict of plain values.  ``listed()`` holds the fixed ones, ``draw(rng)`` gives others of the same
ranges, ``prepare`` makes what a program holds before the call, ``run`` is one pass, ``exact`` the same pass in
64 bits in plain torch.  Sizes are those of the repository's presets and of the files under ``configs/``.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from kolmogorov_moe_architecture_b200 import AdvancedMoEConfig, ops
from kolmogorov_moe_architecture_b200.models.layers import TransformerBlock
from kolmogorov_moe_architecture_b200.models.mamba import MambaBlock
from kolmogorov_moe_architecture_b200.training.losses import MultiTokenPredictionLoss

DEV = "cuda"
BF16 = torch.bfloat16
W_LB, W_Z = 0.01, 0.001                      # auxiliary loss weights of every preset
HEAD_WEIGHTS = (1.0, 0.5, 0.3, 0.2)          # multi-token loss weights of every preset


def listed():
    return [
        # Attention of the 5B preset in a training step: micro-batch 4, full context.
        dict(name="attention-train-5b", op="attention", batch=4, seq=2048, heads=16, kv_heads=4, head_dim=128, docs=0, train=True),
        # Packed documents at an odd length on 64-wide heads (the 500M recipe): what a data loader that packs gives.
        dict(name="attention-train-packed-d64", op="attention", batch=8, seq=1021, heads=12, kv_heads=3, head_dim=64, docs=4, train=True),
        # One prompt of no particular length, forward only: every layer of every generation step.
        dict(name="attention-eval-prompt", op="attention", batch=1, seq=777, heads=12, kv_heads=3, head_dim=128, docs=0, train=False),
        # A whole attention + dense FFN layer in training: norms, projections, rotary embedding, attention, SwiGLU (1.5B recipe).
        dict(name="dense-layer-train", op="layer", batch=4, seq=1024, d=1536, heads=12, kv_heads=3, head_dim=128, ff=4096, train=True),
        # Selective-scan layer of the 5B preset in training.
        dict(name="mamba-train-5b", op="mamba", batch=4, seq=2048, d=2048, train=True),
        # A short odd-length prompt through the selective-scan layer of the 500M recipe, forward only.
        dict(name="mamba-eval-prompt", op="mamba", batch=1, seq=333, d=768, train=False),
        # Routing and experts of the 5B preset in training: 4 x 2048 positions of which depth routing keeps 3/4.
        dict(name="moe-train-5b", op="moe", tokens=6144, d=2048, ff=2816, experts=16, top_k=2, train=True),
        # A short prompt through the experts of the 1.5B recipe, forward only: weights are all there is to read.
        dict(name="moe-eval-prompt", op="moe", tokens=93, d=1536, ff=2048, experts=8, top_k=2, train=False),
        # The 3B preset: 64 experts whose width is no multiple of 64, depth routing keeps half of 4 x 2048.
        dict(name="moe-train-3b-64-experts", op="moe", tokens=4096, d=1792, ff=2464, experts=64, top_k=2, train=True),
        # Expert choice as in the production recipe.
        dict(name="expert-choice-train", op="expert_choice", batch=4, seq=1536, d=2048, ff=2048, experts=16, train=True),
        # Output heads and loss with the vocabulary that most recipes use (1.5B recipe).
        dict(name="loss-train-vocab-50257", op="loss", batch=4, seq=1024, d=1536, vocab=50257, heads=4),
        # Optimizer: orthogonalisation of the stacked Mamba output projections of the 5B preset.
        dict(name="muon-8x2048x4096", op="muon", count=8, rows=2048, cols=4096),
    ]


# ------------------------------------------------------------------ drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["attention", "attention", "layer", "mamba", "moe", "moe", "expert_choice", "loss", "muon"])
    train = rng.random() < 0.7
    if op == "attention":
        heads, kv = rng.choice([(16, 4), (12, 3), (8, 4), (8, 2), (14, 2), (4, 1)])
        seq = _log_int(rng, 33, 2048)
        batch = rng.randint(1, max(1, min(8, 8192 // seq)))
        docs = rng.choice([0, 0, 3, 6]) if seq >= 256 else 0
        return dict(op=op, batch=batch, seq=seq, heads=heads, kv_heads=kv, head_dim=rng.choice([64, 128, 128]), docs=docs,
                    train=train)
    if op == "layer":
        d, heads, kv, hd, ff = rng.choice([(1536, 12, 3, 128, 4096), (1024, 8, 4, 128, 4096), (768, 12, 3, 64, 2048),
                                           (512, 8, 2, 64, 1408), (2048, 16, 4, 128, 5632)])
        seq = _log_int(rng, 33, 1024)
        return dict(op=op, batch=rng.randint(1, max(1, min(4, 4096 // seq))), seq=seq, d=d, heads=heads, kv_heads=kv,
                    head_dim=hd, ff=ff, train=train)
    if op == "mamba":
        seq = _log_int(rng, 33, 2048)
        return dict(op=op, batch=rng.randint(1, max(1, min(4, 8192 // seq))), seq=seq, d=rng.choice([512, 768, 1536, 1792, 2048]),
                    train=train)
    if op == "moe":
        d, ff, experts, top_k = rng.choice([(2048, 2816, 16, 2), (1536, 2048, 8, 2), (1792, 2464, 64, 2), (1792, 2304, 14, 2),
                                            (1024, 4096, 8, 4), (2048, 2560, 12, 2), (1920, 1280, 32, 4), (768, 1024, 8, 2)])
        return dict(op=op, tokens=_log_int(rng, 17, 6144), d=d, ff=ff, experts=experts, top_k=top_k, train=train)
    if op == "expert_choice":
        d, ff, experts = rng.choice([(2048, 2048, 16), (1024, 4096, 8), (1536, 2048, 8)])
        seq = _log_int(rng, 65, 2048)
        return dict(op=op, batch=rng.randint(1, max(1, min(4, 6144 // seq))), seq=seq, d=d, ff=ff, experts=experts, train=train)
    if op == "loss":
        seq = _log_int(rng, 65, 1024)
        return dict(op=op, batch=rng.randint(1, max(1, min(4, 4096 // seq))), seq=seq, d=rng.choice([512, 768, 1024, 1536]),
                    vocab=rng.choice([32000, 50257, 50257, 50304]), heads=rng.choice([2, 4]))
    rows = rng.choice([160, 512, 768, 1024, 1536, 2048])
    cols = rng.choice([1024, 1408, 1536, 2048, 4096, 5632])
    rows, cols = (rows, cols) if rng.random() < 0.5 else (cols, rows)
    return dict(op="muon", count=rng.randint(1, 12), rows=rows, cols=cols)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape, scale=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def _uniform(g, *shape, bound):
    return ((torch.rand(*shape, generator=g, device=DEV) * 2 - 1) * bound).to(BF16)


def _doc_start(g, batch, seq, docs):
    """First position of the document of each position: ``docs`` documents per row, cut at uniform places."""
    cuts = torch.rand(batch, docs - 1, generator=g, device=DEV).mul(seq - 1).long() + 1
    start = torch.zeros(batch, seq, dtype=torch.long, device=DEV)
    start.scatter_(1, cuts, cuts)
    return torch.cummax(start, dim=1).values.to(torch.int32)


def _config(case):
    """One-layer configurations around the layer of a case."""
    kw = dict(vocab_size=32000, n_layers=1, moe_layers=(), mod_enabled=False, dropout=0.0, attention_dropout=0.0,
              residual_dropout=0.0, n_experts=8)
    if case["op"] == "layer":
        return AdvancedMoEConfig(d_model=case["d"], n_heads=case["heads"], n_kv_heads=case["kv_heads"],
                                 head_dim=case["head_dim"], d_ff=case["ff"], mamba_layers=(), **kw)
    return AdvancedMoEConfig(d_model=case["d"], n_heads=case["d"] // 128, n_kv_heads=1, head_dim=128, mamba_layers=(0,), **kw)


def _module(case, seed):
    torch.manual_seed(seed)
    with torch.device(DEV):
        cfg = _config(case)
        m = TransformerBlock(cfg, 0) if case["op"] == "layer" else MambaBlock(cfg)
    return m.to(BF16).train(case["train"])


def prepare(case, seed):
    g, op = _gen(seed), case["op"]
    train = case.get("train", True)
    s = {"case": case, "train": train}
    if op == "attention":
        B, S, H, KV, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        s["leaves"] = [_randn(g, B, S, n, D) for n in (H, KV, KV)]
        s["doc_start"] = _doc_start(g, B, S, case["docs"]) if case["docs"] else None
        s["grad"] = _randn(g, B, S, H, D) if train else None
    elif op in ("layer", "mamba"):
        B, S, d = case["batch"], case["seq"], case["d"]
        m = _module(case, seed)
        s["module"] = m
        # a layer reads the residual stream, a mixer reads normalised rows
        x = _randn(g, B, S, d)
        s["leaves"] = [x] + list(m.parameters())
        s["grad"] = _randn(g, B, S, d) if train else None
    elif op == "moe":
        T, d, f, E, k = (case[n] for n in ("tokens", "d", "ff", "experts", "top_k"))
        x = _randn(g, T, d)
        # loads of a trained router are uneven: Zipf(1)
        logits = (torch.randn(T, E, generator=g, device=DEV) - torch.log(torch.arange(1, E + 1, device=DEV).float())).to(BF16)
        s["leaves"] = [x, logits, _uniform(g, E, d, f, bound=d ** -0.5), _uniform(g, E, d, f, bound=d ** -0.5),
                       _uniform(g, E, f, d, bound=f ** -0.5)]
        s["grad"] = _randn(g, T, d) if train else None
    elif op == "expert_choice":
        B, S, d, f, E = (case[n] for n in ("batch", "seq", "d", "ff", "experts"))
        s["leaves"] = [_randn(g, B, S, d), torch.randn(B, S, E, generator=g, device=DEV), _uniform(g, E, d, f, bound=d ** -0.5),
                       _uniform(g, E, d, f, bound=d ** -0.5), _uniform(g, E, f, d, bound=f ** -0.5)]
        s["capacity"] = min(S, math.ceil(1.25 * S / E))
        s["grad"] = _randn(g, B, S, d) if train else None
    elif op == "loss":
        B, S, d, V, n = (case[k] for k in ("batch", "seq", "d", "vocab", "heads"))
        s["leaves"] = [_randn(g, B, S, d)] + [_randn(g, V, d, scale=0.02) for _ in range(n)]
        labels = torch.randint(0, V, (B, S), generator=g, device=DEV)
        s["labels"] = labels.masked_fill(torch.rand(B, S, generator=g, device=DEV) < 0.05, -100)      # padding
        s["loss"] = MultiTokenPredictionLoss(n, HEAD_WEIGHTS[:n])
    else:
        x = _randn(g, case["count"], case["rows"], case["cols"], scale=1e-3)
        s["leaves"] = [x]
        s["sumsq"] = x.float().square().sum(dim=(1, 2))
        s["train"] = False
    for t in s["leaves"]:
        t.requires_grad_(s["train"])
    return s


# ------------------------------------------------------------------ one pass
def _forward(s):
    case, leaves = s["case"], s["leaves"]
    op = case["op"]
    if op == "attention":
        return (ops.attention(*leaves, causal=True, doc_start=s["doc_start"]),)
    if op in ("layer", "mamba"):
        return (s["module"](leaves[0]),)
    if op == "moe":
        x, logits, w1, w2, w3 = leaves
        w, idx, aux, _counts = ops.route_topk(logits, case["top_k"], W_LB, W_Z)
        return ops.grouped_swiglu(x, w1, w2, w3, idx, w), aux
    if op == "expert_choice":
        x, logits, w1, w2, w3 = leaves
        w, tok = ops.expert_choice_route(logits, s["capacity"])
        return (ops.expert_choice_swiglu(x, w1, w2, w3, w, tok),)
    if op == "loss":
        total, info = s["loss"].from_hidden(leaves[0], leaves[1:], s["labels"])
        return (total,)
    return (ops.newton_schulz(leaves[0], 5, s["sumsq"]),)


def run(s):
    if not s["train"]:
        with torch.no_grad():
            return _forward(s)
    outs = _forward(s)
    seeds = [s["grad"]] if s.get("grad") is not None else [torch.ones_like(outs[0])]
    seeds += [torch.ones_like(o) for o in outs[1:]]
    return (*[o.detach() for o in outs], *torch.autograd.grad(outs, s["leaves"], seeds))


# ------------------------------------------------------------------ the same in 64 bits
def _exact_attention(q, k, v, doc_start):
    B, S, H, D = q.shape
    rep = H // k.shape[2]
    pos = torch.arange(S, device=q.device)
    outs = []
    for b in range(B):
        hidden = pos[None, :] > pos[:, None]
        if doc_start is not None:
            hidden = hidden | (pos[None, :] < doc_start[b].long()[:, None])
        qb = q[b].transpose(0, 1)
        kb, vb = (t[b].transpose(0, 1).repeat_interleave(rep, dim=0) for t in (k, v))
        p = torch.softmax((qb @ kb.transpose(1, 2) / math.sqrt(D)).masked_fill(hidden, float("-inf")), dim=-1)
        outs.append((p @ vb).transpose(0, 1))
    return torch.stack(outs)


def _exact_norm(x, w, eps=1e-5):
    return w * x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _exact_layer(case, x, p):
    B, S, d = x.shape
    H, KV, D = case["heads"], case["kv_heads"], case["head_dim"]
    angle = torch.outer(torch.arange(S, device=x.device).float(), 1.0 / (10000.0 ** (torch.arange(0, D, 2, device=x.device).float() / D)))
    cos, sin = (t.to(BF16).double()[None, :, None, :] for t in (angle.cos(), angle.sin()))    # the layer keeps bf16 tables

    def rope(t):
        a, b = t.chunk(2, dim=-1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)
    h = _exact_norm(x, p["seq_norm.weight"])
    q, k, v = (F.linear(h, p[f"seq_layer.{n}_proj.weight"]).view(B, S, -1, D) for n in "qkv")
    o = _exact_attention(rope(q), rope(k), v, None).reshape(B, S, H * D)
    x = x + F.linear(o, p["seq_layer.o_proj.weight"])
    h = _exact_norm(x, p["ffn_norm.weight"])
    return x + F.linear(F.silu(F.linear(h, p["ffn.w1.weight"])) * F.linear(h, p["ffn.w2.weight"]), p["ffn.w3.weight"])


def _exact_mamba(x, p):
    B, S, d = x.shape
    u, z = F.linear(x, p["mamba.in_proj.weight"]).chunk(2, dim=-1)
    C = u.shape[-1]
    w = p["mamba.conv1d.weight"].squeeze(1)                                   # (C, 4)
    padded = F.pad(u, (0, 0, 3, 0))
    u = F.silu(sum(padded[:, j:j + S] * w[:, j] for j in range(4)) + p["mamba.conv1d.bias"])
    R = p["mamba.dt_proj.weight"].shape[1]
    dt, Bm, Cm = torch.split(F.linear(u, p["mamba.x_proj.weight"]), [R, 16, 16], dim=-1)
    dt = F.softplus(F.linear(dt, p["mamba.dt_proj.weight"]) + p["mamba.dt_proj.bias"])
    A = -torch.exp(p["mamba.A_log"])
    h = torch.zeros(B, C, 16, dtype=x.dtype, device=x.device)
    ys = []
    for t in range(S):
        h = torch.exp(dt[:, t, :, None] * A) * h + (dt[:, t] * u[:, t])[..., None] * Bm[:, t, None, :]
        ys.append(torch.einsum("bcn,bn->bc", h, Cm[:, t]))
    y = (torch.stack(ys, dim=1) + u * p["mamba.D"]) * F.silu(z)
    return F.linear(y, p["mamba.out_proj.weight"])


def _exact_moe(case, x, logits, w1, w2, w3):
    T, E = logits.shape
    k = case["top_k"]
    idx = torch.sort(logits, dim=-1, descending=True, stable=True).indices[:, :k]
    p = torch.softmax(logits, dim=-1)
    w = p.gather(1, idx)
    w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(E):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        y = (F.silu(x[tok] @ w1[e]) * (x[tok] @ w2[e])) @ w3[e]
        out = out.index_add(0, tok, y * w[tok, slot].unsqueeze(1))
    share = torch.bincount(idx.reshape(-1), minlength=E).to(x.dtype) / (T * k)
    aux = W_LB * E * (share * p.mean(0)).sum() + W_Z * torch.logsumexp(logits, dim=-1).square().mean()
    return out, aux


def _exact_choice(capacity, x, logits, w1, w2, w3):
    B, S, d = x.shape
    p = torch.softmax(logits, dim=1).transpose(1, 2)                          # (B, E, S)
    w, tok = torch.topk(p, capacity, dim=-1)
    w = w / (w.sum(-1, keepdim=True) + 1e-9)
    outs = []
    for b in range(B):
        out = torch.zeros_like(x[b])
        for e in range(logits.shape[2]):
            r = x[b, tok[b, e]]
            out = out.index_add(0, tok[b, e], ((F.silu(r @ w1[e]) * (r @ w2[e])) @ w3[e]) * w[b, e, :, None])
        outs.append(out)
    return torch.stack(outs)


def _exact_loss(hidden, heads, labels):
    n = len(heads)
    total = 0.0
    for i, W in enumerate(heads):
        lg = F.linear(hidden[:, : hidden.shape[1] - i - 1], W)
        ce = F.cross_entropy(lg.reshape(-1, lg.shape[-1]), labels[:, i + 1:].reshape(-1), ignore_index=-100)
        total = total + HEAD_WEIGHTS[i] / sum(HEAD_WEIGHTS[:n]) * ce
    return total


def exact(case, seed):
    s = prepare(case, seed)
    op = case["op"]
    leaves = [t.detach().double().requires_grad_(s["train"]) for t in s["leaves"]]
    with torch.set_grad_enabled(s["train"]):
        if op == "attention":
            outs = (_exact_attention(*leaves, s["doc_start"]),)
        elif op in ("layer", "mamba"):
            p = dict(zip([n for n, _ in s["module"].named_parameters()], leaves[1:]))
            outs = (_exact_layer(case, leaves[0], p) if op == "layer" else _exact_mamba(leaves[0], p),)
        elif op == "moe":
            outs = _exact_moe(case, *leaves)
        elif op == "expert_choice":
            outs = (_exact_choice(s["capacity"], *leaves),)
        elif op == "loss":
            outs = (_exact_loss(leaves[0], leaves[1:], s["labels"]),)
        else:
            y = leaves[0] / (leaves[0].flatten(1).norm(dim=1).view(-1, 1, 1) + 1e-7)
            for _ in range(5):
                gram = y @ y.transpose(1, 2) @ y if case["rows"] <= case["cols"] else y @ (y.transpose(1, 2) @ y)
                y = 1.5 * y - 0.5 * gram
            outs = (y,)
    if not s["train"]:
        return tuple(o.detach() for o in outs)
    seeds = [s["grad"].double()] if s.get("grad") is not None else [torch.ones_like(outs[0])]
    seeds += [torch.ones_like(o) for o in outs[1:]]
    return (*[o.detach() for o in outs], *torch.autograd.grad(outs, leaves, seeds))


# ------------------------------------------------------------------ work and tolerance
def work(case):
    op, train = case["op"], case.get("train", True)
    if op == "attention":
        B, S, H, KV, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        pairs = S * S / (case["docs"] + 1) if case["docs"] else S * S / 2       # uniform cuts: sum of squares is 2 S^2 / (docs + 1)
        io = 2.0 * B * S * D
        return {"flops": 4.0 * B * H * pairs * D * (3.5 if train else 1),
                "bytes": io * (2 * H + 2 * KV) + (io * (2 * H + 2 * KV) if train else 0)}
    if op == "layer":
        B, S, d, f = case["batch"], case["seq"], case["d"], case["ff"]
        params = d * (2 * case["heads"] + 2 * case["kv_heads"]) * case["head_dim"] + 3 * d * f
        return {"flops": 2.0 * B * S * params * (3 if train else 1) + 2.0 * B * S * S * d * (3.5 if train else 1),
                "bytes": 2.0 * params * (2 if train else 1) + 2.0 * B * S * d * (4 if train else 2)}
    if op == "mamba":
        B, S, d = case["batch"], case["seq"], case["d"]
        C, R = 2 * d, math.ceil(d / 16)
        params = d * 2 * C + C * (R + 32) + R * C + C * d
        return {"flops": (2.0 * params + 6.0 * 16 * C) * B * S * (3 if train else 1),
                "bytes": 2.0 * params * (2 if train else 1) + 2.0 * B * S * d * (4 if train else 2)}
    if op in ("moe", "expert_choice"):
        d, f, E = case["d"], case["ff"], case["experts"]
        if op == "moe":
            T = case["tokens"]
            rows = T * case["top_k"]
        else:
            T = case["batch"] * case["seq"]
            rows = case["batch"] * E * min(case["seq"], math.ceil(1.25 * case["seq"] / E))
        return {"flops": 6.0 * rows * d * f * (3 if train else 1),
                "bytes": 6.0 * min(E, rows) * d * f * (2 if train else 1) + 2.0 * T * d * (4 if train else 2)}
    if op == "loss":
        T, d, V, n = case["batch"] * case["seq"], case["d"], case["vocab"], case["heads"]
        return {"flops": 6.0 * T * d * V * n, "bytes": 4.0 * n * V * d + 4.0 * T * d}
    b, m, n = case["count"], case["rows"], case["cols"]
    g, o = min(m, n), max(m, n)
    # five steps on the short side (two Gram-sized products a step), or step by step where that is less
    return {"flops": 2.0 * b * min(g * g * o * 1.5 + 6.0 * g ** 3, 7.5 * g * g * o), "bytes": 4.0 * b * m * n}


#: About four times the largest error against 64 bits that was measured for each kind of pass (bf16 operands and
#: results, 32-bit sums): 0.0025, 0.006, 0.007, 0.005, 0.0041, 0.0037, 0.0042 in this order.
_REL = {"attention": 0.01, "layer": 0.024, "mamba": 0.028, "moe": 0.02, "expert_choice": 0.016, "loss": 0.015, "muon": 0.016}


def tolerance(case):
    return {"rel": _REL[case["op"]]}
