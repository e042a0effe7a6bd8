"""The work that programs have this package do, as cases that can be timed and checked one by one.

Every case is one pass of a layer or a model through the public entry points (``piper_b200.ops``, ``piper_b200.nn``,
``piper_b200.models``) on one GPU, in bf16 as the kernels take it.  ``kind`` selects the path:

* ``attention``   causal grouped-query attention on a packed qkv projection, with or without its backward pass
* ``attn_block``  the attention layer: qkv projection, QK-norm, rotary embedding, attention, output projection
* ``ffn``         the SwiGLU MLP; ``sinks`` accumulates weight gradients into fp32 buckets as the executor does
* ``norm``        residual add + RMSNorm
* ``moe``         router, dispatch, grouped expert MLP, combine
* ``head``        output projection + cross-entropy over a large vocabulary
* ``llama``       a whole Llama forward and backward from tokens to logits, loss and weight gradients

Sizes are those of the bundled model configurations, with token counts from 128 to a full 4096- or 8192-token
microbatch, ragged ones among them.  Attention needs sequence lengths that are multiples of 128.
"""
from __future__ import annotations

import math

import torch

from piper_b200 import ops
from piper_b200.models.llama3 import LlamaConfig, Transformer
from piper_b200.nn import Attention, FeedForward, cross_entropy_loss
from piper_b200.ops import moe as moe_ops

BF16 = torch.bfloat16


def listed() -> list:
    return [
        # one microbatch of the 8B configuration: the layer's attention in a training step
        {"name": "attn_8b_train", "kind": "attention", "B": 1, "S": 4096, "Hq": 32, "Hkv": 8, "hd": 128, "grad": True},
        # scoring a long sequence with the 30B-A3B head layout: forward only, the largest sequence
        {"name": "attn_long_fwd", "kind": "attention", "B": 1, "S": 8192, "Hq": 32, "Hkv": 4, "hd": 128, "grad": False},
        # the 1B configuration's 64-wide heads on a batch whose length is no power of two
        {"name": "attn_hd64_train", "kind": "attention", "B": 3, "S": 1408, "Hq": 32, "Hkv": 8, "hd": 64, "grad": True},
        # the 30B-A3B attention layer (QK-norm, half-split rotary) on two 2048-token sequences
        {"name": "block_qwen_train", "kind": "attn_block", "B": 2, "S": 2048, "dim": 2048, "Hq": 32, "Hkv": 4, "hd": 128,
         "qk_norm": True, "interleaved": False},
        # the attention layer of the tiny configuration, the smallest training call: latency and launches
        {"name": "block_tiny_train", "kind": "attn_block", "B": 4, "S": 128, "dim": 256, "Hq": 4, "Hkv": 4, "hd": 64,
         "qk_norm": False, "interleaved": True},
        # the MLP of the 8B configuration in a training step, weight gradients into fp32 buckets
        {"name": "ffn_8b_train", "kind": "ffn", "T": 4096, "dim": 4096, "hidden": 14336, "sinks": True},
        # the MLP of the 3B configuration on a ragged token count, plain autograd
        {"name": "ffn_3b_ragged", "kind": "ffn", "T": 1000, "dim": 3072, "hidden": 8192, "sinks": False},
        # residual add + norm between the two halves of an 8B layer
        {"name": "norm_8b_train", "kind": "norm", "T": 4096, "D": 4096},
        # the expert layer of the 30B-A3B configuration on one microbatch
        {"name": "moe_30b_train", "kind": "moe", "T": 4096, "D": 2048, "E": 128, "k": 8, "F": 768},
        # the expert layer of the 1B mixture on a ragged token count: small segments
        {"name": "moe_1b_ragged", "kind": "moe", "T": 777, "D": 1024, "E": 32, "k": 4, "F": 512},
        # output projection and loss of the 1B configuration on one microbatch with padded labels
        {"name": "head_1b_train", "kind": "head", "T": 4096, "D": 2048, "V": 128256},
        # a whole (shallow) model of the 1B configuration's widths: embedding to loss and back
        {"name": "llama_1b_2layer", "kind": "llama", "B": 2, "S": 1024, "layers": 2, "dim": 2048, "Hq": 32, "Hkv": 8,
         "hidden": 8192, "V": 128256},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["attention", "attention", "attn_block", "ffn", "ffn", "norm", "moe", "moe", "head", "llama"])
    if kind == "attention":
        hd = rng.choice([64, 128])
        Hkv = rng.choice([2, 4, 8])
        Hq = Hkv * rng.choice([1, 2, 4, 8] if Hkv <= 4 else [1, 2, 4])
        S = 128 * _log_int(rng, 1, 40)
        B = _log_int(rng, 1, max(1, 8192 // S))
        return {"kind": kind, "B": B, "S": S, "Hq": Hq, "Hkv": Hkv, "hd": hd, "grad": rng.random() < 0.7}
    if kind == "attn_block":
        hd = rng.choice([64, 128])
        Hkv = rng.choice([2, 4, 8])
        Hq = Hkv * rng.choice([1, 2, 4])
        S = 128 * _log_int(rng, 1, 24)
        B = _log_int(rng, 1, max(1, 4096 // S))
        qwen = rng.random() < 0.5
        return {"kind": kind, "B": B, "S": S, "dim": rng.choice([256, 1024, 2048, 3072, 4096]), "Hq": Hq, "Hkv": Hkv,
                "hd": hd, "qk_norm": qwen, "interleaved": not qwen}
    if kind == "ffn":
        dim, hidden = rng.choice([(256, 688), (256, 768), (2048, 8192), (3072, 8192), (4096, 14336), (2048, 6144)])
        return {"kind": kind, "T": _log_int(rng, 100, 4096), "dim": dim, "hidden": hidden, "sinks": rng.random() < 0.5}
    if kind == "norm":
        return {"kind": kind, "T": _log_int(rng, 100, 8192), "D": rng.choice([256, 1024, 2048, 2560, 3072, 4096, 8192])}
    if kind == "moe":
        D, E, k, F = rng.choice([(256, 8, 2, 256), (1024, 32, 4, 512), (2048, 64, 8, 768), (2048, 128, 8, 768)])
        return {"kind": kind, "T": _log_int(rng, 128, 4096), "D": D, "E": E, "k": k, "F": F}
    if kind == "head":
        return {"kind": kind, "T": _log_int(rng, 100, 4096), "D": rng.choice([256, 1024, 2048]),
                "V": rng.choice([1024, 2048, 32000, 128256])}
    dim, Hq, Hkv, hidden = rng.choice([(256, 4, 4, 688), (1024, 16, 4, 4096), (2048, 32, 8, 8192)])
    S = 128 * _log_int(rng, 1, 12)
    return {"kind": kind, "B": _log_int(rng, 1, max(1, 2048 // S)), "S": S, "layers": rng.choice([1, 2]), "dim": dim,
            "Hq": Hq, "Hkv": Hkv, "hidden": hidden, "V": rng.choice([1024, 2048, 32000])}


# ------------------------------------------------------------------ inputs
def _llama_config(c: dict) -> LlamaConfig:
    return LlamaConfig(dim=c["dim"], n_layers=c["layers"], n_heads=c["Hq"], n_kv_heads=c["Hkv"], vocab_size=c["V"],
                       ffn_hidden=c["hidden"], max_seq_len=c["S"])


def _inputs(c: dict, seed: int) -> dict:
    """Every tensor of a case, made from the seed alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rn(*shape, std=1.0):
        return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * std).to(BF16)

    kind = c["kind"]
    if kind == "attention":
        T = c["B"] * c["S"]
        t = {"qkv": rn(T, (c["Hq"] + 2 * c["Hkv"]) * c["hd"])}
        if c["grad"]:
            t["dout"] = rn(T, c["Hq"] * c["hd"])
        return t
    if kind == "attn_block":
        T, dim, hd = c["B"] * c["S"], c["dim"], c["hd"]
        t = {"x": rn(T, dim), "wqkv": rn((c["Hq"] + 2 * c["Hkv"]) * hd, dim, std=dim ** -0.5),
             "wo": rn(dim, c["Hq"] * hd, std=(c["Hq"] * hd) ** -0.5), "dout": rn(T, dim)}
        if c["qk_norm"]:
            t["qw"] = 1.0 + rn(hd, std=0.1)
            t["kw"] = 1.0 + rn(hd, std=0.1)
        return t
    if kind == "ffn":
        T, dim, F = c["T"], c["dim"], c["hidden"]
        return {"x": rn(T, dim), "w13": rn(2 * F, dim, std=dim ** -0.5), "w2": rn(dim, F, std=F ** -0.5),
                "dout": rn(T, dim)}
    if kind == "norm":
        T, D = c["T"], c["D"]
        return {"x": rn(T, D), "res": rn(T, D), "w": 1.0 + rn(D, std=0.1), "dy": rn(T, D), "dh": rn(T, D)}
    if kind == "moe":
        T, D, E, F = c["T"], c["D"], c["E"], c["F"]
        # Logits without ties, so that the selection is a property of the inputs: every row holds the quantiles of a
        # normal distribution, in an order that favours some experts over others, as a router in training does.
        quant = torch.special.ndtri((torch.arange(E, dtype=torch.float64) + 0.5) / E).float().cuda()
        bias = torch.randn(E, generator=g, device="cuda") * 0.3
        rank = (torch.randn(T, E, generator=g, device="cuda") + bias).argsort(1).argsort(1)
        return {"x": rn(T, D), "logits": quant[rank].to(BF16), "w13": rn(E, 2 * F, D, std=D ** -0.5),
                "w2": rn(E, D, F, std=F ** -0.5), "dout": rn(T, D)}
    if kind == "head":
        T, D, V = c["T"], c["D"], c["V"]
        labels = torch.randint(0, V, (T,), generator=g, device="cuda")
        labels[torch.rand(T, generator=g, device="cuda") < 0.03] = -100
        return {"x": rn(T, D), "w": rn(V, D, std=D ** -0.5), "labels": labels}
    t = {"tokens": torch.randint(0, c["V"], (c["B"], c["S"]), generator=g, device="cuda"),
         "labels": torch.randint(0, c["V"], (c["B"], c["S"]), generator=g, device="cuda")}
    with torch.device("meta"):
        shapes = {n: p.shape for n, p in Transformer(_llama_config(c), c["S"], 1).named_parameters()}
    for n, shape in shapes.items():
        t[n] = 1.0 + rn(*shape, std=0.1) if len(shape) == 1 else rn(*shape, std=1.0 if "embed" in n else shape[1] ** -0.5)
    return t


def _fill(module: torch.nn.Module, values: dict) -> torch.nn.Module:
    module = module.to_empty(device="cuda").to(BF16)
    with torch.no_grad():
        for n, p in module.named_parameters():
            p.copy_(values[n])
    return module


def prepare(case: dict, seed: int) -> dict:
    c, t = case, _inputs(case, seed)
    s = {"case": c}
    kind = c["kind"]
    if kind == "attn_block":
        with torch.device("meta"):
            m = Attention(c["dim"], c["Hq"], c["Hkv"], c["hd"], qk_norm=c["qk_norm"], rope_interleaved=c["interleaved"])
        vals = {"wqkv.weight": t["wqkv"], "wo.weight": t["wo"]}
        if c["qk_norm"]:
            vals.update({"q_norm.weight": t["qw"], "k_norm.weight": t["kw"]})
        s["module"] = _fill(m, vals)
        s["cos"], s["sin"] = ops.rope_tables(c["hd"], c["S"], 500000.0, device="cuda")
        s["x"], s["dout"] = t["x"].requires_grad_(True), t["dout"]
    elif kind == "ffn":
        with torch.device("meta"):
            m = FeedForward(c["dim"], c["hidden"])
        s["module"] = _fill(m, {"w13.weight": t["w13"], "w2.weight": t["w2"]})
        s["x"], s["dout"] = t["x"].requires_grad_(True), t["dout"]
        if c["sinks"]:
            s["sinks"] = [torch.empty(p.shape, dtype=torch.float32, device="cuda") for p in m.parameters()]
    elif kind == "llama":
        cfg = _llama_config(c)
        with torch.device("meta"):
            m = Transformer(cfg, c["S"], 1)
        m = _fill(m, t)
        k = Transformer.const_attrs(cfg, c["S"], "cuda")
        m.rope_cos, m.rope_sin = k["rope_cos"], k["rope_sin"]
        s["module"], s["tokens"], s["labels"] = m, t["tokens"], t["labels"]
    else:
        s.update({n: v.requires_grad_(v.is_floating_point() and not n.startswith("d")) for n, v in t.items()})
    return s


def run(s: dict):
    c = s["case"]
    kind = c["kind"]
    if kind == "attention":
        if not c["grad"]:
            with torch.no_grad():
                return ops.attention(s["qkv"], c["B"], c["S"], c["Hq"], c["Hkv"], c["hd"])
        out = ops.attention(s["qkv"], c["B"], c["S"], c["Hq"], c["Hkv"], c["hd"])
        (dqkv,) = torch.autograd.grad(out, s["qkv"], s["dout"])
        # the three gradients apart: dK and dV are small beside dQ in some layouts, large in others
        nq, nk = c["Hq"] * c["hd"], c["Hkv"] * c["hd"]
        return {"out": out, "dq": dqkv[:, :nq], "dk": dqkv[:, nq:nq + nk], "dv": dqkv[:, nq + nk:]}
    if kind == "attn_block":
        m = s["module"]
        out = m(s["x"], s["cos"], s["sin"], c["B"], c["S"])
        names = ["x"] + [n for n, _ in m.named_parameters()]
        grads = torch.autograd.grad(out, [s["x"], *m.parameters()], s["dout"])
        return {"out": out, **{"d" + n: v for n, v in zip(names, grads)}}
    if kind == "ffn":
        m = s["module"]
        if not c["sinks"]:
            out = m(s["x"])
            dx, dw13, dw2 = torch.autograd.grad(out, [s["x"], m.w13.weight, m.w2.weight], s["dout"])
            return {"out": out, "dx": dx, "dw13": dw13, "dw2": dw2}
        for p, sink in zip(m.parameters(), s["sinks"]):
            sink.zero_()                       # the first microbatch of a step starts from cleared buckets
            ops.grad_sinks.register(p, sink)
        try:
            out = m(s["x"])
            dx = torch.autograd.grad(out, [s["x"], *m.parameters()], s["dout"], allow_unused=True)[0]
        finally:
            for p in m.parameters():
                ops.grad_sinks.unregister(p)
        return {"out": out, "dx": dx, "dw13": s["sinks"][0], "dw2": s["sinks"][1]}
    if kind == "norm":
        y, h = ops.add_rmsnorm(s["x"], s["res"], s["w"], 1e-5)
        dx, dw = torch.autograd.grad([y, h], [s["x"], s["w"]], [s["dy"], s["dh"]])
        return {"y": y, "h": h, "dx": dx, "dw": dw}
    if kind == "moe":
        weights, idx, counts = moe_ops.moe_route(s["logits"], c["k"], True)
        rows, pos, g_start, g_len, ep_counts = moe_ops.moe_dispatch(s["x"], idx, counts)
        gs, gl = moe_ops.moe_group_table(ep_counts, s["w13"])
        h = moe_ops.grouped_linear(rows, s["w13"], gs, gl)
        o = moe_ops.grouped_linear(ops.swiglu(h), s["w2"], gs, gl)
        out = moe_ops.moe_combine(o, pos, weights, g_start, g_len, counts)
        dx, dlogits, dw13, dw2 = torch.autograd.grad(out, [s["x"], s["logits"], s["w13"], s["w2"]], s["dout"])
        return {"out": out, "dx": dx, "dlogits": dlogits, "dw13": dw13, "dw2": dw2}
    if kind == "head":
        loss = ops.cross_entropy(ops.linear(s["x"], s["w"]), s["labels"])
        dx, dw = torch.autograd.grad(loss, [s["x"], s["w"]])
        return {"loss": loss, "dx": dx, "dw": dw}
    m = s["module"]
    logits = m(s["tokens"])
    loss = cross_entropy_loss(logits, s["labels"])
    grads = torch.autograd.grad(loss, list(m.parameters()))
    return {"logits": logits, "loss": loss, **{"d" + n: v for (n, _), v in zip(m.named_parameters(), grads)}}


# -------------------------------------------------------- what a pass costs
def _attn_flops(B, S, Hq, hd, grad) -> float:
    fwd = 4.0 * B * Hq * hd * S * (S + 1) / 2
    return fwd * (3.5 if grad else 1.0)          # backward: S, dP, dV, dQ, dK against S and PV


def work(case: dict) -> dict:
    c = case
    kind = c["kind"]
    if kind == "attention":
        T, W, O = c["B"] * c["S"], (c["Hq"] + 2 * c["Hkv"]) * c["hd"], c["Hq"] * c["hd"]
        by = 2.0 * T * (W + O) + (2.0 * T * (O + W) if c["grad"] else 0.0)
        return {"bytes": by, "flops": _attn_flops(c["B"], c["S"], c["Hq"], c["hd"], c["grad"])}
    if kind == "attn_block":
        T, W, O, D = c["B"] * c["S"], (c["Hq"] + 2 * c["Hkv"]) * c["hd"], c["Hq"] * c["hd"], c["dim"]
        return {"bytes": 2.0 * (4 * T * D + 2 * W * D + 2 * D * O),
                "flops": 6.0 * T * D * (W + O) + _attn_flops(c["B"], c["S"], c["Hq"], c["hd"], True)}
    if kind == "ffn":
        T, D, F = c["T"], c["dim"], c["hidden"]
        return {"bytes": 2.0 * 4 * T * D + 3.0 * F * D * (2 + (4 if c["sinks"] else 2)), "flops": 18.0 * T * D * F}
    if kind == "norm":
        return {"bytes": 2.0 * 7 * c["T"] * c["D"], "flops": 12.0 * c["T"] * c["D"]}
    if kind == "moe":
        T, D, E, k, F = c["T"], c["D"], c["E"], c["k"], c["F"]
        return {"bytes": 2.0 * (4 * T * D + 2 * T * E + 2 * 3 * E * F * D), "flops": 18.0 * T * k * D * F}
    if kind == "head":
        T, D, V = c["T"], c["D"], c["V"]
        return {"bytes": 2.0 * (2 * T * D + 2 * V * D) + 8.0 * T, "flops": 6.0 * T * D * V}
    T, D, F, V, L = c["B"] * c["S"], c["dim"], c["hidden"], c["V"], c["layers"]
    kv = D // c["Hq"] * c["Hkv"]
    per = D * (D + 2 * kv) + D * D + 3 * F * D
    return {"bytes": 2.0 * (2 * (L * per + 2 * V * D) + T * V) + 16.0 * T,
            "flops": 6.0 * T * (L * per + V * D) + L * _attn_flops(c["B"], c["S"], c["Hq"], D // c["Hq"], True)}


def tolerance(case: dict) -> dict:
    """bf16 operands and results with fp32 accumulation; about four times the distance from the 64-bit result."""
    return {"rel": {"attention": 1e-2, "attn_block": 2.5e-2, "ffn": 1.4e-2, "norm": 1e-2, "moe": 1.7e-2, "head": 1.7e-2,
                    "llama": 4e-2}[case["kind"]]}


# ------------------------------------------------------------- 64-bit results
def _attn64(qkv, B, S, Hq, Hkv, hd):
    """[T, (Hq + 2 Hkv) hd] fp64 -> [T, Hq hd], one kv group at a time."""
    x = qkv.view(B, S, Hq + 2 * Hkv, hd)
    r = Hq // Hkv
    mask = torch.ones(S, S, dtype=torch.bool, device=qkv.device).triu(1)
    rows = []
    for b in range(B):
        heads = []
        for g in range(Hkv):
            q = x[b, :, g * r:(g + 1) * r].transpose(0, 1)
            p = torch.softmax((q @ x[b, :, Hq + g].t() / math.sqrt(hd)).masked_fill(mask, float("-inf")), dim=-1)
            heads.append((p @ x[b, :, Hq + Hkv + g]).transpose(0, 1))
        rows.append(torch.cat(heads, dim=1))
    return torch.stack(rows).reshape(B * S, Hq * hd)


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _rope64(qkv, S, Hq, Hkv, hd, interleaved, qw, kw, eps):
    T = qkv.shape[0]
    cos, sin = ops.rope_tables(hd, S, 500000.0, device="cuda")
    pos = torch.arange(T, device="cuda") % S
    cs, sn = cos.double()[pos].unsqueeze(1), sin.double()[pos].unsqueeze(1)
    x = qkv.view(T, Hq + 2 * Hkv, hd)
    parts = []
    for t, w in ((x[:, :Hq], qw), (x[:, Hq:Hq + Hkv], kw)):
        if w is not None:
            t = _norm64(t, w, eps)
        a, b = (t[..., 0::2], t[..., 1::2]) if interleaved else (t[..., :hd // 2], t[..., hd // 2:])
        u, v = a * cs - b * sn, a * sn + b * cs
        parts.append(torch.stack((u, v), -1).flatten(-2) if interleaved else torch.cat((u, v), -1))
    return torch.cat((*parts, x[:, Hq + Hkv:]), dim=1).reshape(T, -1)


def _swiglu64(h):
    g, u = h.chunk(2, dim=-1)
    return torch.nn.functional.silu(g) * u


def exact(case: dict, seed: int):
    c = case
    t = {n: (v.double().requires_grad_(not n.startswith("d")) if v.is_floating_point() else v)
         for n, v in _inputs(case, seed).items()}
    kind = c["kind"]
    if kind == "attention":
        if not c["grad"]:
            with torch.no_grad():
                return _attn64(t["qkv"], c["B"], c["S"], c["Hq"], c["Hkv"], c["hd"])
        out = _attn64(t["qkv"], c["B"], c["S"], c["Hq"], c["Hkv"], c["hd"])
        (d,) = torch.autograd.grad(out, t["qkv"], t["dout"])
        nq, nk = c["Hq"] * c["hd"], c["Hkv"] * c["hd"]
        return {"out": out, "dq": d[:, :nq], "dk": d[:, nq:nq + nk], "dv": d[:, nq + nk:]}
    if kind == "attn_block":
        qkv = _rope64(t["x"] @ t["wqkv"].t(), c["S"], c["Hq"], c["Hkv"], c["hd"], c["interleaved"], t.get("qw"),
                      t.get("kw"), 1e-6)
        out = _attn64(qkv, c["B"], c["S"], c["Hq"], c["Hkv"], c["hd"]) @ t["wo"].t()
        keys = {"x": "x", "wqkv.weight": "wqkv", "wo.weight": "wo"}
        if c["qk_norm"]:
            keys.update({"q_norm.weight": "qw", "k_norm.weight": "kw"})
        grads = torch.autograd.grad(out, [t[v] for v in keys.values()], t["dout"])
        return {"out": out, **{"d" + n: v for n, v in zip(keys, grads)}}
    if kind == "ffn":
        out = _swiglu64(t["x"] @ t["w13"].t()) @ t["w2"].t()
        dx, dw13, dw2 = torch.autograd.grad(out, [t["x"], t["w13"], t["w2"]], t["dout"])
        return {"out": out, "dx": dx, "dw13": dw13, "dw2": dw2}
    if kind == "norm":
        h = t["x"] + t["res"]
        y = _norm64(h, t["w"], 1e-5)
        dx, dw = torch.autograd.grad([y, h], [t["x"], t["w"]], [t["dy"], t["dh"]])
        return {"y": y, "h": h, "dx": dx, "dw": dw}
    if kind == "moe":
        w, idx = torch.topk(torch.softmax(t["logits"], dim=-1), c["k"], dim=-1)
        w = w / w.sum(-1, keepdim=True)
        out = torch.zeros_like(t["x"])
        w13, w2 = t["w13"].unbind(0), t["w2"].unbind(0)
        for e in range(c["E"]):
            tok, slot = (idx == e).nonzero(as_tuple=True)
            o = _swiglu64(t["x"][tok] @ w13[e].t()) @ w2[e].t()
            out = out.index_add(0, tok, o * w[tok, slot].unsqueeze(-1))
        grads = torch.autograd.grad(out, [t["x"], t["logits"], t["w13"], t["w2"]], t["dout"])
        return {"out": out, **dict(zip(("dx", "dlogits", "dw13", "dw2"), grads))}
    if kind == "head":
        loss = torch.nn.functional.cross_entropy(t["x"] @ t["w"].t(), t["labels"])
        dx, dw = torch.autograd.grad(loss, [t["x"], t["w"]])
        return {"loss": loss, "dx": dx, "dw": dw}
    names = [n for n in t if n not in ("tokens", "labels")]
    hd, eps = c["dim"] // c["Hq"], 1e-5
    h = t["tok_embeddings.weight"][t["tokens"].reshape(-1)]
    for i in range(c["layers"]):
        p = f"layers.{i}."
        qkv = _norm64(h, t[p + "attention_norm.weight"], eps) @ t[p + "attention.wqkv.weight"].t()
        qkv = _rope64(qkv, c["S"], c["Hq"], c["Hkv"], hd, True, None, None, eps)
        h = h + _attn64(qkv, c["B"], c["S"], c["Hq"], c["Hkv"], hd) @ t[p + "attention.wo.weight"].t()
        y = _norm64(h, t[p + "ffn_norm.weight"], eps)
        h = h + _swiglu64(y @ t[p + "feed_forward.w13.weight"].t()) @ t[p + "feed_forward.w2.weight"].t()
    logits = (_norm64(h, t["norm.weight"], eps) @ t["output.weight"].t()).view(c["B"], c["S"], c["V"])
    loss = torch.nn.functional.cross_entropy(logits.view(-1, c["V"]), t["labels"].reshape(-1))
    grads = torch.autograd.grad(loss, [t[n] for n in names])
    return {"logits": logits, "loss": loss, **{"d" + n: v for n, v in zip(names, grads)}}
