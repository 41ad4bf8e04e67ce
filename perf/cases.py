"""Performance cases: what a reinforcement-learning program has this framework do.

One GRPO step is rollout (a decode step per token, then a draw from the logits), scoring of the
finished sequences, the loss, and backward through the model. Every case is one of those pieces
called through its public entry point at the sizes such a program meets: a Llama-3-8B-shaped
model (hidden 4096, 32 query heads over 8 KV heads, FFN 14336, vocabulary 128256), 512 tokens
per sequence, 8 to 256 sequences; ``draw`` adds other sizes of the same ranges, odd ones among them.
"""
from __future__ import annotations

import math

import torch

from kernel_align_b200.kernels.sampling import SamplerBackend
from kernel_align_b200.models.llama import DecoderLayer, LlamaConfig
from kernel_align_b200.ops.attention import attention_fn
from kernel_align_b200.ops.decode import attention_decode, decode_qkv_rope_cache
from kernel_align_b200.ops.fused_logp import lmhead_logp
from kernel_align_b200.ops.gemm import gemm_bi
from kernel_align_b200.ops.grpo_loss import group_advantages, grpo_loss
from kernel_align_b200.ops.layer_ops import rmsnorm, rope_tables, swiglu
from kernel_align_b200.ops.logits_logp import logits_logp
from kernel_align_b200.parallel.tp_gemm import TPContext

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_8B = {"hidden": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336}
_SMALL = {"hidden": 1024, "heads": 8, "kv_heads": 2, "ffn": 4096}
_HEAD_DIM = 128
_EPS = 1e-5
_THETA = 500000.0


def listed():
    return [
        # the loss of one policy update: 64 completions of 384 tokens, group advantages, clipped
        # ratio, k3 KL to a reference policy, and the gradient for the log-probs: the smallest call
        {"name": "grpo_loss_64x384", "kind": "grpo", "seqs": 64, "length": 384, "group": 8, "mask": True, "ref": True,
         "seq_mean": False},
        # the draw of one decode step with the usual filters
        {"name": "sample_topk_64", "kind": "sample", "rows": 64, "vocab": 128256, "dtype": "bf16", "top_k": 50,
         "top_p": 0.9, "temperature": 0.7},
        # nucleus sampling without top-k for a large batch of sequences
        {"name": "sample_topp_200", "kind": "sample", "rows": 200, "vocab": 128256, "dtype": "bf16", "top_k": 0,
         "top_p": 0.9, "temperature": 1.0},
        # scoring of tokens from logits that another engine has produced (the reference's API)
        {"name": "logits_logp_2048", "kind": "logits_logp", "rows": 2048, "vocab": 128256, "dtype": "bf16"},
        # scoring of 32 finished sequences under the old or the reference policy, from hidden states
        {"name": "lmhead_logp_16384", "kind": "lmhead", "rows": 16384, "hidden": 4096, "vocab": 128256, "train": False},
        # the policy's log-probs with gradients for one micro-batch of ragged completions
        {"name": "lmhead_logp_train_2000", "kind": "lmhead", "rows": 2000, "hidden": 4096, "vocab": 128256,
         "train": True},
        # attention of a training micro-batch, forward and backward
        {"name": "attention_train_8x512", "kind": "attention", "batch": 8, "length": 512, "heads": 32, "kv_heads": 8,
         "causal": True},
        # the same for long sequences whose length is no multiple of a tile
        {"name": "attention_train_2x4000", "kind": "attention", "batch": 2, "length": 4000, "heads": 32, "kv_heads": 8,
         "causal": True},
        # one decoder layer of a decode step, as it is replayed from a graph for every new token:
        # a handful of sequences, and a whole group of rollouts
        {"name": "decode_layer_8x512", "kind": "decode", "batch": 8, "cache": 512, **_8B},
        {"name": "decode_layer_64x1000", "kind": "decode", "batch": 64, "cache": 1000, **_8B},
        # one decoder layer in a scoring pass over a single sequence (no gradients)
        {"name": "layer_forward_1x512", "kind": "layer", "batch": 1, "length": 512, "train": False, **_8B},
        # one decoder layer of a training micro-batch, forward and backward
        {"name": "layer_train_8x512", "kind": "layer", "batch": 8, "length": 512, "train": True, **_8B},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grpo", "sample", "sample", "logits_logp", "lmhead", "lmhead", "attention", "attention", "decode",
                       "decode", "layer", "layer"])
    if kind == "grpo":
        group = rng.choice([2, 4, 8, 16])
        return {"kind": kind, "seqs": group * _log_int(rng, 4, 16), "length": _log_int(rng, 33, 1024), "group": group,
                "mask": rng.random() < 0.7, "ref": rng.random() < 0.5, "seq_mean": rng.random() < 0.3}
    if kind == "sample":
        top_k = rng.choice([0, 0, 1, 20, 50, 200, 1000])
        return {"kind": kind, "rows": _log_int(rng, 1, 256), "vocab": rng.choice([32000, 50257, 128256, 128255]),
                "dtype": rng.choice(["bf16", "bf16", "bf16", "fp32", "fp16"]), "top_k": top_k,
                "top_p": rng.choice([1.0, 0.9, 0.95]), "temperature": rng.choice([0.7, 1.0])}
    if kind == "logits_logp":
        return {"kind": kind, "rows": _log_int(rng, 8, 2048), "vocab": rng.choice([32000, 50257, 128256]),
                "dtype": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "lmhead":
        train = rng.random() < 0.5
        return {"kind": kind, "rows": _log_int(rng, 100, 2000 if train else 16384), "hidden": rng.choice([1024, 2048, 4096]),
                "vocab": rng.choice([32000, 50304, 128256]), "train": train}
    if kind == "attention":
        heads, kv_heads = rng.choice([(32, 8), (8, 2), (16, 16), (4, 1)])
        length = _log_int(rng, 64, 4000)
        return {"kind": kind, "batch": max(1, min(8, rng.randint(1, 8000 // length))), "length": length, "heads": heads,
                "kv_heads": kv_heads, "causal": rng.random() < 0.8}
    if kind == "decode":
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "cache": _log_int(rng, 60, 1500),
                **(_8B if rng.random() < 0.7 else _SMALL)}
    length = _log_int(rng, 50, 1024)
    return {"kind": "layer", "batch": rng.randint(1, max(1, 4096 // length)), "length": length,
            "train": rng.random() < 0.6, **(_8B if rng.random() < 0.6 else _SMALL)}


# ---- inputs ---------------------------------------------------------------------------------


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _normal(gen, *shape, std=1.0, dtype=torch.bfloat16):
    out = torch.empty(*shape, dtype=dtype, device=_device())
    flat = out.view(-1)
    step = 1 << 28
    for i in range(0, flat.numel(), step):
        n = min(step, flat.numel() - i)
        flat[i:i + n] = torch.randn(n, device=_device(), generator=gen) * std
    return out


def _weights(case, gen):
    h, hq, hkv, f = case["hidden"], case["heads"], case["kv_heads"], case["ffn"]
    return {"wqkv": _normal(gen, (hq + 2 * hkv) * _HEAD_DIM, h, std=0.02), "wo": _normal(gen, h, hq * _HEAD_DIM, std=0.02),
            "wgu": _normal(gen, 2 * f, h, std=0.02), "wdown": _normal(gen, h, f, std=0.02),
            "norm1": _normal(gen, h, std=0.1) + 1, "norm2": _normal(gen, h, std=0.1) + 1}


def _inputs(case, seed):
    """The tensors of a case, from the seed alone (shared by ``prepare`` and ``exact``)."""
    gen, dev, kind = _gen(seed), _device(), case["kind"]
    if kind == "grpo":
        shape = (case["seqs"], case["length"])
        old = -(torch.rand(shape, device=dev, generator=gen) * 3)
        new = old + torch.randn(shape, device=dev, generator=gen) * 0.15
        ref = old + torch.randn(shape, device=dev, generator=gen) * 0.1
        ends = torch.randint(case["length"] // 2, case["length"] + 1, (case["seqs"], 1), device=dev, generator=gen)
        mask = (torch.arange(case["length"], device=dev)[None] < ends).float()
        return {"new": new, "old": old, "ref": ref if case["ref"] else None, "mask": mask if case["mask"] else None,
                "rewards": torch.randn(case["seqs"], device=dev, generator=gen)}
    if kind in ("sample", "logits_logp"):
        logits = _normal(gen, case["rows"], case["vocab"], std=2.0, dtype=_DTYPES[case["dtype"]])
        return {"logits": logits, "ids": torch.randint(0, case["vocab"], (case["rows"],), device=dev, generator=gen)}
    if kind == "lmhead":
        d = {"hidden": _normal(gen, case["rows"], case["hidden"]),
             "weight": _normal(gen, case["vocab"], case["hidden"], std=0.02),
             "ids": torch.randint(0, case["vocab"], (case["rows"],), device=dev, generator=gen)}
        if case["train"]:
            d["grad"] = torch.randn(case["rows"], device=dev, generator=gen) / case["rows"]
        return d
    if kind == "attention":
        b, l = case["batch"], case["length"]
        return {"q": _normal(gen, b, l, case["heads"], _HEAD_DIM), "k": _normal(gen, b, l, case["kv_heads"], _HEAD_DIM),
                "v": _normal(gen, b, l, case["kv_heads"], _HEAD_DIM), "grad": _normal(gen, b, l, case["heads"], _HEAD_DIM)}
    w = _weights(case, gen)
    if kind == "decode":
        b, t = case["batch"], case["cache"]
        shape = (b, t, case["kv_heads"], _HEAD_DIM)
        return {**w, "x": _normal(gen, b, case["hidden"]), "delta": _normal(gen, b, case["hidden"]),
                "cache_k": _normal(gen, *shape), "cache_v": _normal(gen, *shape), "pos": t - t // 8 - 1}
    rows = -(-case["batch"] * case["length"] // 128) * 128
    x = torch.zeros(rows, case["hidden"], dtype=torch.bfloat16, device=dev)
    tokens = case["batch"] * case["length"]
    x[:tokens] = _normal(gen, tokens, case["hidden"])
    d = {**w, "x": x}
    if case["train"]:
        g = torch.zeros_like(x)
        g[:tokens] = _normal(gen, tokens, case["hidden"])
        d["grad"] = g
    return d


def _decode_step(s):
    h, x = rmsnorm(s["delta"], s["norm1"], _EPS, residual=s["x"])
    qkv = gemm_bi(h, s["wqkv"])
    q = decode_qkv_rope_cache(qkv, s["pos_t"], s["slot"], s["cos"], s["sin"], s["cache_k"], s["cache_v"], s["heads"],
                              s["kv_heads"])
    a = attention_decode(q, s["cache_k"], s["cache_v"], s["lens"]).reshape(x.shape[0], -1)
    h, x = rmsnorm(gemm_bi(a, s["wo"]), s["norm2"], _EPS, residual=x)
    return x, gemm_bi(swiglu(gemm_bi(h, s["wgu"])), s["wdown"]), s["cache_k"], s["cache_v"]


def prepare(case, seed):
    s = {"case": case, **_inputs(case, seed)}
    kind, dev = case["kind"], _device()
    if kind == "grpo":
        s["new"].requires_grad_(True)
    elif kind == "sample":
        s["sampler"] = SamplerBackend(seed=int(seed) & 0xFFFF)
    elif kind == "lmhead" and case["train"]:
        s["hidden"].requires_grad_(True)
        s["weight"].requires_grad_(True)
    elif kind == "attention":
        for n in ("q", "k", "v"):
            s[n].requires_grad_(True)
    elif kind == "decode":
        # a serving loop keeps position, length and slot on the device and replays one graph per token
        b, pos = case["batch"], s["pos"]
        s["cos"], s["sin"] = rope_tables(case["cache"], _HEAD_DIM, _THETA, device=dev)
        s["pos_t"] = torch.full((b,), pos, dtype=torch.int64, device=dev)
        s["lens"] = torch.full((b,), pos + 1, dtype=torch.int32, device=dev)
        s["slot"] = torch.full((1,), pos, dtype=torch.int64, device=dev)
        s["heads"], s["kv_heads"] = case["heads"], case["kv_heads"]
        _decode_step(s)                      # loads every kernel before the capture
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = _decode_step(s)
    elif kind == "layer":
        cfg = LlamaConfig(hidden=case["hidden"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], head_dim=_HEAD_DIM,
                          ffn=case["ffn"], n_layers=1, rope_theta=_THETA, rms_eps=_EPS)
        layer = DecoderLayer(cfg, TPContext(device=dev), 1, dev)
        layer.load_state_dict({n: s.pop(n) for n, _ in layer.named_parameters()}, assign=True)
        s["layer"] = layer.requires_grad_(case["train"])
        s["positions"] = torch.arange(case["length"], device=dev).repeat(case["batch"])
        s["cos"], s["sin"] = rope_tables(case["length"], _HEAD_DIM, _THETA, device=dev)
        s["x"].requires_grad_(case["train"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "grpo":
        adv = group_advantages(s["rewards"], case["group"])
        loss = grpo_loss(s["new"], s["old"], adv, mask=s["mask"], logp_ref=s["ref"], beta=0.04 if case["ref"] else 0.0,
                         reduction="seq_mean" if case["seq_mean"] else "token_mean")
        return loss.detach(), torch.autograd.grad(loss, s["new"])[0]
    if kind == "sample":
        return s["sampler"].sample(s["logits"], top_k=case["top_k"] or None,
                                   top_p=case["top_p"] if case["top_p"] < 1 else None, temperature=case["temperature"], step=3)
    if kind == "logits_logp":
        return logits_logp(s["logits"], s["ids"])
    if kind == "lmhead":
        logp = lmhead_logp(s["hidden"], s["weight"], s["ids"])
        if not case["train"]:
            return logp
        return (logp.detach(), *torch.autograd.grad(logp, (s["hidden"], s["weight"]), s["grad"]))
    if kind == "attention":
        out = attention_fn(s["q"], s["k"], s["v"], causal=case["causal"])
        return (out.detach(), *torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["grad"]))
    if kind == "decode":
        s["graph"].replay()
        return s["out"]
    with torch.set_grad_enabled(case["train"]):
        y = s["layer"](s["x"], case["batch"], case["length"], s["positions"], s["cos"], s["sin"])
    if not case["train"]:
        return y
    return (y.detach(), *torch.autograd.grad(y, (s["x"], *s["layer"].parameters()), s["grad"]))


# ---- what a pass cannot do without -----------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "grpo":
        n = case["seqs"] * case["length"]
        return {"bytes": n * 4 * (3 + bool(case["ref"]) + bool(case["mask"])) + case["seqs"] * 4, "flops": 20 * n}
    if kind in ("sample", "logits_logp"):
        n = case["rows"] * case["vocab"]
        return {"bytes": n * (4 if case["dtype"] == "fp32" else 2) + case["rows"] * 12, "flops": 3 * n}
    if kind == "lmhead":
        m, k, v = case["rows"], case["hidden"], case["vocab"]
        once = (m + v) * k * 2
        return {"bytes": once * (2 if case["train"] else 1) + 12 * m, "flops": 2 * m * k * v * (3 if case["train"] else 1)}
    if kind == "attention":
        b, l, hq, hkv = case["batch"], case["length"], case["heads"], case["kv_heads"]
        pairs = b * hq * l * (l + 1) // 2 if case["causal"] else b * hq * l * l
        # in: q, k, v and the incoming gradient; out: the result and three gradients
        return {"bytes": b * l * _HEAD_DIM * 2 * (4 * hq + 4 * hkv), "flops": 2 * _HEAD_DIM * pairs * (2 + 5)}
    h, hq, hkv, f = case["hidden"], case["heads"], case["kv_heads"], case["ffn"]
    wn = (hq + 2 * hkv) * _HEAD_DIM * h + h * hq * _HEAD_DIM + 3 * h * f
    if kind == "decode":
        b, n = case["batch"], case["cache"] - case["cache"] // 8
        return {"bytes": 2 * wn + b * n * hkv * _HEAD_DIM * 4 + 8 * b * h,
                "flops": 2 * b * wn + 4 * b * n * hq * _HEAD_DIM}
    b, l = case["batch"], case["length"]
    t = b * l
    pairs = b * hq * l * (l + 1) // 2
    if not case["train"]:
        return {"bytes": 2 * wn + 4 * t * h, "flops": 2 * t * wn + 4 * _HEAD_DIM * pairs}
    return {"bytes": 4 * wn + 8 * t * h, "flops": 6 * t * wn + 2 * _HEAD_DIM * pairs * 7}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return "exact"           # integer arithmetic after a fixed exponential: the same token for the same stream
    # about four times the distance from ``exact`` that was measured
    if kind == "grpo":
        return {"rel": 1e-6}             # 1.8e-7: sums in 32 bits
    if kind == "logits_logp":
        return {"rel": 5e-7}             # 3.8e-8 in 128256 columns, up to 1e-7 in fewer
    if kind == "lmhead":
        return {"rel": 1e-2} if case["train"] else {"rel": 3e-6}     # 2.4e-3 (bf16 gradients) and 7e-7
    if kind == "attention":
        return {"rel": 1e-2}             # 2.5e-3: probabilities and results in bf16
    if kind == "decode":
        return {"rel": 2.5e-2}           # 6.4e-3: bf16 between nine kernels
    return {"rel": 4e-2}                 # 1.1e-2: bf16 between the kernels of a layer, both directions


# ---- the same in 64 bits ---------------------------------------------------------------------


def _attend(q, k, v, causal):
    """softmax(q k^T / sqrt(d)) v for ``[B, L, H, D]``, KV heads repeated over their group."""
    g = q.shape[2] // k.shape[2]
    qh, kh, vh = q.transpose(1, 2), k.transpose(1, 2).repeat_interleave(g, 1), v.transpose(1, 2).repeat_interleave(g, 1)
    outs = []
    for i in range(0, qh.shape[1], 8):          # a few heads at a time
        sc = qh[:, i:i + 8] @ kh[:, i:i + 8].transpose(-1, -2) / math.sqrt(q.shape[-1])
        if causal:
            n = sc.shape[-1]
            sc = sc.masked_fill(torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1), -math.inf)
        outs.append(torch.softmax(sc, -1) @ vh[:, i:i + 8])
    return torch.cat(outs, 1).transpose(1, 2)


def _norm(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + _EPS) * w


def _rotate(x, cos, sin):
    a, b = x[..., : _HEAD_DIM // 2], x[..., _HEAD_DIM // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _exact_layer(case, d):
    b, l, hq, hkv, f = case["batch"], case["length"], case["heads"], case["kv_heads"], case["ffn"]
    t = b * l
    cos, sin = (c.double()[None, :, None] for c in rope_tables(l, _HEAD_DIM, _THETA, device=_device()))
    x = d["x"]
    qkv = (_norm(x, d["norm1"]) @ d["wqkv"].t())[:t].view(b, l, hq + 2 * hkv, _HEAD_DIM)
    a = _attend(_rotate(qkv[:, :, :hq], cos, sin), _rotate(qkv[:, :, hq:hq + hkv], cos, sin), qkv[:, :, hq + hkv:], True)
    a = torch.cat([a.reshape(t, -1), a.new_zeros(x.shape[0] - t, hq * _HEAD_DIM)])
    x = x + a @ d["wo"].t()
    gu = _norm(x, d["norm2"]) @ d["wgu"].t()
    return x + (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ d["wdown"].t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None
    d = {k: v.double() if isinstance(v, torch.Tensor) and v.is_floating_point() else v for k, v in _inputs(case, seed).items()}
    if kind == "grpo":
        new = d["new"].requires_grad_(True)
        r = d["rewards"].view(-1, case["group"])
        adv = ((r - r.mean(1, keepdim=True)) / (r.std(1, keepdim=True) + 1e-4)).view(-1, 1)
        ratio = torch.exp(new - d["old"])
        tok = -torch.minimum(ratio * adv, ratio.clamp(0.8, 1.2) * adv)
        if case["ref"]:
            dr = d["ref"] - new
            tok = tok + 0.04 * (torch.exp(dr) - dr - 1)
        m = d["mask"] if case["mask"] else torch.ones_like(tok)
        loss = ((tok * m).sum(1) / m.sum(1)).mean() if case["seq_mean"] else (tok * m).sum() / m.sum()
        return loss.detach(), torch.autograd.grad(loss, new)[0]
    if kind == "logits_logp":
        return torch.log_softmax(d["logits"], -1).gather(1, d["ids"][:, None])[:, 0]
    if kind == "lmhead":
        logp, dh, dw = [], [], None
        for i in range(0, case["rows"], 2048):
            h, ids = d["hidden"][i:i + 2048], d["ids"][i:i + 2048, None]
            lg = torch.log_softmax(h @ d["weight"].t(), -1)
            logp.append(lg.gather(1, ids)[:, 0])
            if case["train"]:
                g = d["grad"][i:i + 2048, None]
                dl = lg.exp_().mul_(-g).scatter_add_(1, ids, g)
                dh.append(dl @ d["weight"])
                dw = dl.t() @ h if dw is None else dw + dl.t() @ h
        return (torch.cat(logp), torch.cat(dh), dw) if case["train"] else torch.cat(logp)
    if kind == "attention":
        q, k, v = (d[n].requires_grad_(True) for n in ("q", "k", "v"))
        outs, grads = [], []
        for i in range(case["batch"]):
            o = _attend(q[i:i + 1], k[i:i + 1], v[i:i + 1], case["causal"])
            grads.append(torch.autograd.grad(o, (q, k, v), d["grad"][i:i + 1]))
            outs.append(o.detach())
        return (torch.cat(outs), *(sum(g[n] for g in grads) for n in range(3)))
    if kind == "decode":
        b, hq, hkv, f, pos = case["batch"], case["heads"], case["kv_heads"], case["ffn"], d["pos"]
        cos, sin = (c.double()[pos] for c in rope_tables(case["cache"], _HEAD_DIM, _THETA, device=_device()))
        x = d["x"] + d["delta"]
        qkv = (_norm(x, d["norm1"]) @ d["wqkv"].t()).view(b, hq + 2 * hkv, _HEAD_DIM)
        ck, cv = d["cache_k"], d["cache_v"]
        ck[:, pos], cv[:, pos] = _rotate(qkv[:, hq:hq + hkv], cos, sin), qkv[:, hq + hkv:]
        q = _rotate(qkv[:, :hq], cos, sin)[:, None]
        a = _attend(q, ck[:, : pos + 1], cv[:, : pos + 1], False).reshape(b, -1)
        x = x + a @ d["wo"].t()
        gu = _norm(x, d["norm2"]) @ d["wgu"].t()
        return x, (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ d["wdown"].t(), ck, cv
    if not case["train"]:
        with torch.no_grad():
            return _exact_layer(case, d)
    names = ("x", "wqkv", "wo", "wgu", "wdown", "norm1", "norm2")
    leaves = [d[n].requires_grad_(True) for n in names]
    y = _exact_layer(case, d)
    return (y.detach(), *torch.autograd.grad(y, leaves, d["grad"]))
