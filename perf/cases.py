"""Workloads that stand for what users of this package run: the quantised expert FFN of a mixture-of-experts layer, operator
by operator and as a whole, from one small call to a full prefill batch.

The layer is: ``moe_init_routing_v3`` (tokens grouped by expert and quantised per row), ``grouped_matmul_swiglu_quant``
(gate/up GEMM, SwiGLU, requantisation), ``grouped_matmul_v4`` (down GEMM, one row per (token, slot) pair) or
``grouped_matmul_finalize_routing`` (down GEMM with the weighted sum into token rows).  Model-sized cases use the sizes of
``synth.CONFIGS`` (hidden 7168, intermediate 2048, top-8); int8 operands are rounded normal values with a standard deviation
of about 32 (what per-row quantisation makes of activations and weights), scales give pre-activations of order one, routing
is the top-k of normal logits or a Zipf draw.
"""
from __future__ import annotations

import math

import torch

import ops_transformer_b200 as ops

DEV = "cuda:0"


def listed():
    return [
        # the smallest real call: one gate/up GEMM of a small model, a few hundred rows; latency and launches
        dict(name="gate_up_small", op="swiglu", tokens=64, top_k=4, experts=4, skew=0.0, K=1024, N=2048, fmt="nd"),
        # decoding with 128 sequences: 1024 rows over 256 skewed experts, the weights stream from memory once
        dict(name="gate_up_decode", op="swiglu", tokens=128, top_k=8, experts=256, skew=1.1, K=7168, N=4096, fmt="nd"),
        # the down projection of the same step, with the weights in the storage format that callers of the reference hold
        dict(name="down_decode_nz", op="gmm", tokens=128, top_k=8, experts=256, skew=1.1, K=2048, N=7168, fmt="nz", out="bf16"),
        # prefill of 4096 tokens on a rank with 32 experts, both weight formats
        dict(name="gate_up_prefill", op="swiglu", tokens=4096, top_k=8, experts=32, skew=0.0, K=7168, N=4096, fmt="nd"),
        dict(name="gate_up_prefill_nz", op="swiglu", tokens=4096, top_k=8, experts=32, skew=0.0, K=7168, N=4096, fmt="nz"),
        # the down projection of that prefill, one bf16 row per (token, slot) pair
        dict(name="down_prefill", op="gmm", tokens=4096, top_k=8, experts=32, skew=0.0, K=2048, N=7168, fmt="nd", out="bf16"),
        # the same with the weighted sum into the token rows on top of the shared expert's rows (this operator takes NZ)
        dict(name="down_combine_prefill", op="finalize", tokens=4096, top_k=8, experts=32, skew=0.0, K=2048, N=7168),
        # a middling batch with sizes that fill no tile: bias, GELU and an fp16 result, transposed weight view
        dict(name="down_ragged_bias_gelu", op="gmm", tokens=611, top_k=5, experts=13, skew=0.6, K=1424, N=2976, fmt="trans",
             out="f16", bias=True, act=2),
        # routing and per-row quantisation in front of the prefill
        dict(name="routing_prefill", op="routing", tokens=4096, top_k=8, experts=32, skew=0.0, h=7168, dtype="bf16", smooth=False,
             first=0, last=32),
        # routing of a decoding step on a rank that owns 64 of 256 experts, with per-expert smoothing scales
        dict(name="routing_decode_smooth", op="routing", tokens=128, top_k=8, experts=256, skew=0.0, h=7168, dtype="f16", smooth=True,
             first=64, last=128),
        # the whole layer, decoding with 16 sequences on a small model: four dependent operators, launch bound
        dict(name="layer_decode", op="layer", tokens=16, top_k=8, experts=64, skew=0.0, h=2048, inter=768),
        # the whole layer on a medium batch of the large model
        dict(name="layer_prefill", op="layer", tokens=1000, top_k=8, experts=32, skew=0.0, h=7168, inter=2048),
    ]


def _span(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Sizes over the range of the listed cases: 1 to 4096 tokens, 2 to 256 experts, widths of 256 to 8192 in steps of 16
    or 32; never more operations than the largest prefill nor more weight bytes than the decode case."""
    op = rng.choice(["swiglu", "swiglu", "gmm", "gmm", "finalize", "routing", "layer"])
    while True:
        tokens, experts = _span(rng, 1, 4096), _span(rng, 2, 256)
        top_k = rng.randint(1, min(8, experts))
        skew = rng.choice([0.0, 0.0, 0.6, 1.1])
        if op == "routing":
            first = rng.choice([0, 0, experts // 4])
            return dict(op=op, tokens=tokens, top_k=top_k, experts=experts, skew=skew, h=16 * _span(rng, 16, 512),
                        dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), smooth=rng.random() < 0.3, first=first,
                        last=experts if first == 0 else experts - experts // 4)
        K = 16 * _span(rng, 16, 512)
        N = 64 * _span(rng, 4, 128)
        if 2.0 * tokens * top_k * K * N > 1.9e12 or experts * K * N > 7.5e9:
            continue
        if op == "layer":
            inter = 32 * _span(rng, 8, 128)
            h = 32 * _span(rng, 8, 256)
            if 6.0 * tokens * top_k * h * inter > 1.9e12 or 3 * experts * h * inter > 7.5e9:
                continue
            return dict(op=op, tokens=tokens, top_k=top_k, experts=experts, skew=skew, h=h, inter=inter)
        c = dict(op=op, tokens=tokens, top_k=top_k, experts=experts, skew=skew, K=K, N=N)
        if op == "swiglu":
            c["fmt"] = rng.choice(["nd", "nz"])
        if op == "gmm":
            c["fmt"] = rng.choice(["nd", "nd", "nz", "trans"])
            c["out"] = rng.choice(["bf16", "bf16", "f16", "i32"])
            if c["out"] != "i32" and rng.random() < 0.3:
                c.update(bias=True, act=rng.choice([0, 1, 2, 4, 5]))
        return c


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------

_TORCH = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32, "i32": torch.int32}


def _gen(seed, what):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 64 + what)
    return g


def _routes(case, seed):
    """Expert ids [tokens, top_k] (int32): the top-k of logits plus Gumbel noise (a Zipf draw without replacement) or of
    normal logits."""
    g, n, e = _gen(seed, 0), case["tokens"], case["experts"]
    if case["skew"] > 0:
        u = torch.rand(n, e, device=DEV, generator=g).clamp_(1e-9, 1 - 1e-7)
        logits = -case["skew"] * torch.log(torch.arange(1, e + 1, device=DEV, dtype=torch.float32)) - torch.log(-torch.log(u))
    else:
        logits = torch.randn(n, e, device=DEV, generator=g)
    return logits.topk(case["top_k"], dim=1).indices.to(torch.int32)


def _int8(shape, g):
    out = torch.empty(shape, dtype=torch.int8, device=DEV)
    flat = out.view(-1)
    for i in range(0, flat.numel(), 1 << 26):
        part = flat[i:i + (1 << 26)]
        part.copy_(torch.randn(part.numel(), device=DEV, generator=g).mul_(32).round_().clamp_(-127, 127))
    return out


def _weight(E, K, N, fmt, seed, what):
    """int8 weights in the storage of the format: [E, K, N], the transposed view of [E, N, K], or FRACTAL_NZ."""
    g = _gen(seed, what)
    if fmt == "nz":
        return _int8((E, N // 32, K // 16, 16, 32), g)
    if fmt == "trans":
        return _int8((E, N, K), g).transpose(1, 2)
    return _int8((E, K, N), g)


def _expert(w, e):
    """One expert's weight as [K, N] float64."""
    if w.dim() == 5:
        n1, k1 = w.shape[1], w.shape[2]
        return w[e].permute(1, 2, 0, 3).reshape(k1 * 16, n1 * 32).double()
    return w[e].double()


def _scales(shape, mean, g):
    return torch.empty(shape, device=DEV).uniform_(0.5 * mean, 1.5 * mean, generator=g)


def _counts(case, seed):
    return torch.bincount(_routes(case, seed).view(-1).long(), minlength=case["experts"])


def _inputs(case, seed):
    op, E = case["op"], case["experts"]
    s = {"case": case}
    if op == "routing":
        s["idx"] = _routes(case, seed)
        s["x"] = torch.randn(case["tokens"], case["h"], device=DEV, generator=_gen(seed, 1)).to(_TORCH[case["dtype"]])
        s["smooth"] = _scales((case["last"] - case["first"], case["h"]), 1.0, _gen(seed, 2)) if case["smooth"] else None
        return s
    if op == "layer":
        h, inter = case["h"], case["inter"]
        s["idx"] = _routes(case, seed)
        s["x"] = torch.randn(case["tokens"], h, device=DEV, generator=_gen(seed, 1)).to(torch.bfloat16)
        s["w1"] = _weight(E, h, 2 * inter, "nd", seed, 3)
        s["s1"] = _scales((E, 2 * inter), 1 / (32 * math.sqrt(h)), _gen(seed, 4))
        s["w2"] = _weight(E, inter, h, "nz", seed, 5)
        s["s2"] = _scales((E, h), 1 / (32 * math.sqrt(inter)), _gen(seed, 6))
        logits = torch.rand(case["tokens"], case["top_k"], device=DEV, generator=_gen(seed, 7)) + 0.05
        s["probs"] = (logits / logits.sum(1, keepdim=True)).reshape(-1)
        s["shared"] = torch.randn(case["tokens"], h, device=DEV, generator=_gen(seed, 8)).to(torch.bfloat16)
        return s
    M, K, N = case["tokens"] * case["top_k"], case["K"], case["N"]
    counts = _counts(case, seed)
    s["x"] = _int8((M, K), _gen(seed, 1))
    s["xs"] = _scales((M,), 1 / 32, _gen(seed, 2))
    s["w"] = _weight(E, K, N, case.get("fmt", "nz"), seed, 3)
    s["ws"] = _scales((E, N), 1 / (32 * math.sqrt(K)), _gen(seed, 4))
    s["counts"] = counts
    s["group_list"] = counts if op == "finalize" else counts.cumsum(0)
    if case.get("bias"):
        s["bias"] = torch.randint(-2000, 2000, (E, N), device=DEV, generator=_gen(seed, 5), dtype=torch.int32)
    if op == "finalize":
        pairs = torch.argsort(_routes(case, seed).view(-1).long(), stable=True)
        s["row_index"] = pairs // case["top_k"]
        s["logit"] = torch.rand(M, device=DEV, generator=_gen(seed, 6)) * 0.5 + 0.05
        s["shared"] = torch.randn(case["tokens"], N, device=DEV, generator=_gen(seed, 7)).to(torch.bfloat16)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    if case["op"] == "routing":  # a rank that owns part of the experts leaves rows untouched: the caller's zeroed buffers
        n = case["tokens"] * case["top_k"]
        s["out"] = (torch.zeros(n, case["h"], dtype=torch.int8, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV),
                    torch.zeros(case["last"] - case["first"], dtype=torch.int64, device=DEV), torch.zeros(n, device=DEV))
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    op = case["op"]
    if op == "swiglu":
        fmt = ops.ACL_FORMAT_FRACTAL_NZ if case["fmt"] == "nz" else ops.ACL_FORMAT_ND
        return ops.grouped_matmul_swiglu_quant(s["x"], s["w"], s["ws"], s["xs"], s["group_list"], weight_format=fmt)
    if op == "gmm":
        fmt = ops.ACL_FORMAT_FRACTAL_NZ if case["fmt"] == "nz" else ops.ACL_FORMAT_ND
        i32 = case["out"] == "i32"
        return ops.grouped_matmul_v4(s["x"], s["w"], None if i32 else s["ws"], None if i32 else s["xs"], s["group_list"],
                                     bias=s.get("bias"), act_type=case.get("act", 0), out_dtype=_TORCH[case["out"]],
                                     weight_format=fmt)
    if op == "finalize":
        return ops.grouped_matmul_finalize_routing(s["x"], s["w"], s["ws"], s["group_list"], s["row_index"], case["tokens"],
                                                   pertoken_scale=s["xs"], shared_input=s["shared"], logit=s["logit"])
    if op == "routing":
        return ops.moe_init_routing_v3(s["x"], s["idx"], expert_num=case["experts"],
                                       active_expert_range=(case["first"], case["last"]), quant_mode=1, scale=s["smooth"],
                                       row_idx_type=0, outputs=s["out"])
    E = case["experts"]
    rows, pair_of_row, counts, row_scale = ops.moe_init_routing_v3(s["x"], s["idx"], expert_num=E, active_expert_range=(0, E),
                                                                   quant_mode=1, row_idx_type=1)
    q, qs = ops.grouped_matmul_swiglu_quant(rows, s["w1"], s["s1"], row_scale, counts.cumsum(0))
    pairs = pair_of_row.long()
    y = ops.grouped_matmul_finalize_routing(q, s["w2"], s["s2"], counts, pairs // case["top_k"], case["tokens"],
                                            pertoken_scale=qs, shared_input=s["shared"], logit=s["probs"][pairs])
    return y, counts


# ---------------------------------------------------------------------------------------------------------------------
# work, tolerance and the result in 64 bits
# ---------------------------------------------------------------------------------------------------------------------

def work(case):
    n, k, E = case["tokens"], case["top_k"], case["experts"]
    M, op = n * k, case["op"]
    used = min(E, M) if case["skew"] == 0 else int((_counts(case, 0) > 0).sum())
    if op == "routing":
        active = M * (case["last"] - case["first"]) / E
        size = 4 if case["dtype"] == "f32" else 2
        b = n * case["h"] * size + active * (case["h"] + 8) + M * 8 + (case["last"] - case["first"]) * 8
        if case["smooth"]:
            b += (case["last"] - case["first"]) * case["h"] * 4
        return {"bytes": int(b), "flops": 0}
    if op == "layer":
        h, i = case["h"], case["inter"]
        b = n * h * (2 + 2 + 4) + used * 3 * h * i + used * (2 * i + h) * 4 + M * 12 + E * 8
        return {"bytes": int(b), "flops": int(6 * M * h * i)}
    K, N = case["K"], case["N"]
    b = M * K + used * (K * N + 4 * N) + M * 4 + E * 8
    if op == "swiglu":
        b += M * (N // 2) + M * 4
    elif op == "gmm":
        b += M * N * (4 if case["out"] == "i32" else 2) + (used * N * 4 if case.get("bias") else 0)
    else:
        b += n * N * (4 + 2) + M * 12
    return {"bytes": int(b), "flops": int(2 * M * K * N)}


def tolerance(case):
    op = case["op"]
    if op == "gmm":
        if case["out"] == "i32":
            return "exact"
        # one rounding to the result type: a relative error of up to 2^-9 (bf16) or 2^-12 (fp16) per element
        return {"rel": 5e-3, "max": 1e-2} if case["out"] == "bf16" else {"rel": 6e-4, "max": 1.5e-3}
    if op == "swiglu":  # fp32 chain; an int8 value differs where the scaled value lies on a rounding boundary
        return {"rel": 4e-6, "max": 2e-5, "differ": 2e-4}
    if op == "routing":
        return {"rel": 1e-6, "max": 4e-6, "differ": 2e-5}
    if op == "finalize":  # fp32 sums of at most nine terms in any order
        return {"rel": 2e-6, "max": 4e-5}
    # the layer: single int8 steps of the two requantisations travel through the GEMMs (7e-4 against 64 bits)
    return {"rel": 3e-3, "max": 5e-2}


def _swiglu64(acc, xs, ws):
    v = acc * xs[:, None] * ws[None, :]
    a, b = v.chunk(2, dim=1)
    s = b * (a / (1 + torch.exp(-a)))
    qs = s.abs().amax(1) / 127
    q = (s / qs[:, None]).half().double().round().clamp(-128, 127).to(torch.int8)
    return q, qs


def _act64(kind, v):
    if kind == 1:
        return v.clamp_min(0)
    if kind == 2:
        return v / (1 + torch.exp(-1.59576912 * (v + 0.044715 * v ** 3)))
    if kind == 4:
        return v / (1 + torch.exp(-1.702 * v))
    if kind == 5:
        return v / (1 + torch.exp(-v))
    return v


def _quant64(v):
    """Rows to int8: scale = max / 127, quotient cut to fp16, rounded half away from zero."""
    qs = v.abs().amax(1) / 127
    f = (v / qs[:, None]).nan_to_num(0.0)
    cut = torch.where(f.half().double().abs() > f.abs(), torch.nextafter(f.half(), torch.zeros_like(f.half())), f.half()).double()
    return (torch.sign(cut) * torch.floor(cut.abs() + 0.5)).clamp(-128, 127).to(torch.int8), qs


def _route64(case, s):
    """Output rows in expert order: (pair of every row, its expert, counts)."""
    ids = s["idx"].view(-1).long()
    order = torch.argsort(ids, stable=True)
    return order, ids[order]


def exact(case, seed):
    op, E = case["op"], case["experts"]
    s = _inputs(case, seed)
    if op == "routing":
        first, last, k = case["first"], case["last"], case["top_k"]
        order, ids = _route64(case, s)
        keep = (ids >= first) & (ids < last)
        order, ids = order[keep], ids[keep]
        n = case["tokens"] * k
        rows = torch.zeros(n, case["h"], dtype=torch.int8, device=DEV)
        scale = torch.zeros(n, dtype=torch.float64, device=DEV)
        for i in range(0, order.numel(), 4096):
            v = s["x"][order[i:i + 4096] // k].double()
            if s["smooth"] is not None:
                v = v * s["smooth"][ids[i:i + 4096] - first].double()
            q, qs = _quant64(v)
            rows[i:i + q.shape[0]], scale[i:i + q.shape[0]] = q, qs
        where = torch.full((n,), -1, dtype=torch.int32, device=DEV)
        where[order] = torch.arange(order.numel(), dtype=torch.int32, device=DEV)
        return rows, where, torch.bincount(ids - first, minlength=last - first), scale
    if op == "layer":
        k = case["top_k"]
        order, ids = _route64(case, s)
        counts = torch.bincount(ids, minlength=E)
        y = s["shared"].double()
        at = 0
        for e, c in enumerate(counts.tolist()):
            if c == 0:
                continue
            part = order[at:at + c]
            q, qs = _quant64(s["x"][part // k].double())
            q, qs = _swiglu64(q.double() @ _expert(s["w1"], e), qs, s["s1"][e].double())
            t = (q.double() @ _expert(s["w2"], e)) * qs[:, None] * s["s2"][e].double()[None, :]
            y.index_add_(0, part // k, t * s["probs"][part].double()[:, None])
            at += c
        return y, counts
    counts = s["counts"].tolist()
    M, N = case["tokens"] * case["top_k"], case["N"]
    if op == "swiglu":
        q_all = torch.empty(M, N // 2, dtype=torch.int8, device=DEV)
        qs_all = torch.empty(M, dtype=torch.float64, device=DEV)
    elif op == "finalize":
        y = s["shared"].double()
    else:
        y = torch.empty(M, N, dtype=torch.int32 if case["out"] == "i32" else torch.float64, device=DEV)
    at = 0
    for e, c in enumerate(counts):
        if c == 0:
            continue
        rows = slice(at, at + c)
        acc = s["x"][rows].double() @ _expert(s["w"], e)
        xs, ws = s["xs"][rows].double(), s["ws"][e].double()
        if op == "swiglu":
            q_all[rows], qs_all[rows] = _swiglu64(acc, xs, ws)
        elif op == "finalize":
            y.index_add_(0, s["row_index"][rows], acc * ws[None, :] * xs[:, None] * s["logit"][rows].double()[:, None])
        elif case["out"] == "i32":
            y[rows] = acc.to(torch.int32)
        else:
            if "bias" in s:
                acc = acc + s["bias"][e].double()[None, :]
            y[rows] = _act64(case.get("act", 0), acc * ws[None, :] * xs[:, None])
        at += c
    return (q_all, qs_all) if op == "swiglu" else y
