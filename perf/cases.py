"""The work that a user of this framework has it do, as measurable cases.

Every case goes through a public entry point: the fused route (`ops.route_fused`), the drop-in
select operator (`fused_select_cuda.fused_select_forward`), the Sinkhorn router, the MoE block
(`MoELayer`), the sparse and the dense expert layer on a routing (`strategies.moe_forward`,
`strategies.masked_matmul_forward`) and the drop-in grouped GEMM (`grouped_ffn_cuda`).  The listed
sizes are those of the benchmark (4096 tokens, d_model 4096, hidden 8192, 64 or 8 experts, top 2)
with the decode, long, wide and ragged batches around them; `draw` spreads over the same ranges.
The library is forward-only, so there is no backward direction.
"""
import math
import random

import torch

from moe_routers_b200 import fused_select_cuda, grouped_ffn_cuda, ops, strategies
from moe_routers_b200.moe_layer import MoELayer
from moe_routers_b200.routers import SinkhornRouter

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_ROUTE_OUTPUTS = ("idx", "gates", "counts", "offsets", "packed", "row_route", "route_row")


def listed():
    return [
        # One decode step of a serving batch: 16 tokens routed; launches and host work are all there is.
        dict(name="route_decode", kind="route", tokens=16, d=4096, experts=64, top_k=2, dtype="fp16", skew=False),
        # The benchmark's route: a 4096-token prefill, skewed towards the first 8 experts.
        dict(name="route_prefill", kind="route", tokens=4096, d=4096, experts=64, top_k=2, dtype="fp16", skew=True),
        # A long ragged batch (several sequences packed together) in bf16.
        dict(name="route_long", kind="route", tokens=16387, d=4096, experts=64, top_k=2, dtype="bf16", skew=False),
        # A fine-grained MoE: many experts, many picks per token, odd token count.
        dict(name="route_wide", kind="route", tokens=2049, d=2048, experts=256, top_k=8, dtype="bf16", skew=False),
        # The reference's own operator on given logits: select + count + scan + pack.
        dict(name="select_pack", kind="select_pack", tokens=4096, d=4096, experts=64, top_k=2, dtype="fp16"),
        # The balanced router plug-in on the logits of a prefill batch, 10 iterations.
        dict(name="sinkhorn", kind="sinkhorn", tokens=4096, experts=64, top_k=2, dtype="fp16"),
        # The MoE block in a decode step of 4 sequences: few tokens, the touched experts' weights stream.
        dict(name="layer_decode", kind="layer", tokens=4, d=4096, hidden=8192, experts=64, top_k=2, dtype="fp16"),
        # The MoE block in a ragged bf16 prefill; experts hold a few hundred rows each.
        dict(name="layer_prefill", kind="layer", tokens=2103, d=2048, hidden=5632, experts=32, top_k=4, dtype="bf16"),
        # The benchmark's sparse layer: 64 experts, about 128 rows each as the router deals them.
        dict(name="ffn_64", kind="ffn", tokens=4096, d=4096, hidden=8192, experts=64, top_k=2, dtype="fp16"),
        # The same layer with 8 large experts, about 1024 rows each: bound by the tensor cores.
        dict(name="ffn_8", kind="ffn", tokens=4096, d=4096, hidden=8192, experts=8, top_k=2, dtype="fp16"),
        # The reference's grouped GEMM operator as its demo feeds it: lists of views, [K, N] weights.
        dict(name="grouped_gemm", kind="grouped", tokens=1000, d=4096, hidden=11008, experts=64, top_k=2, dtype="fp16"),
        # Strategy A: every expert over all tokens, gate-masked; the largest amount of arithmetic.
        dict(name="masked_matmul", kind="masked", tokens=4096, d=4096, hidden=8192, experts=8, top_k=2, dtype="fp16"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _multiple(rng, lo, hi, step):
    return min(hi, max(lo, step * round(_log_int(rng, lo, hi) / step)))


def draw(rng):
    kind = rng.choice(["route", "route", "select_pack", "sinkhorn", "layer", "layer", "ffn", "ffn", "grouped", "masked"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind == "route":
        experts = rng.choice([8, 16, 32, 60, 64, 96, 128, 160, 256])
        top_k = rng.choice([1, 2, 2, 4, 6, 8])
        tokens = _log_int(rng, 1, 16384 if top_k <= 2 else 8192)
        # mostly whole 64-wide k blocks; sometimes only the 8 elements that the copies need
        d = _multiple(rng, 512, 8192, 64 if rng.random() < 0.75 else 8)
        return dict(kind=kind, tokens=tokens, d=d, experts=experts, top_k=top_k, dtype=dtype, skew=rng.random() < 0.25)
    if kind == "select_pack":  # the operator's own fixed sizes: 64 experts, top 2, fp16 tokens
        return dict(kind=kind, tokens=_log_int(rng, 1, 16384), d=_multiple(rng, 512, 8192, 64), experts=64, top_k=2, dtype="fp16")
    if kind == "sinkhorn":
        experts = rng.choice([8, 16, 32, 60, 64, 96, 128])
        return dict(kind=kind, tokens=_log_int(rng, 64, 16384), experts=experts, top_k=rng.choice([1, 2, 4]), dtype=dtype)
    d = _multiple(rng, 512, 4096, 64)
    hidden = _multiple(rng, 1024, 8192, 64 if rng.random() < 0.75 else 16)
    if kind == "layer":
        experts = rng.choice([8, 16, 32, 60, 64])
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), d=d, hidden=hidden, experts=experts, top_k=rng.choice([1, 2, 4]), dtype=dtype)
    if kind == "ffn":
        experts = rng.choice([8, 16, 32, 60, 64])
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), d=d, hidden=hidden, experts=experts, top_k=rng.choice([1, 2, 4]), dtype=dtype)
    if kind == "grouped":  # [K, N] weights come in whole 64-column blocks
        experts = rng.choice([8, 16, 32, 64])
        hidden = _multiple(rng, 1024, 11008, 64)
        return dict(kind=kind, tokens=_log_int(rng, 16, 4096), d=d, hidden=hidden, experts=experts, top_k=2, dtype="fp16")
    return dict(kind=kind, tokens=_log_int(rng, 64, 4096), d=d, hidden=hidden, experts=rng.choice([4, 8]), top_k=2, dtype=dtype)


def _randn(gen, shape, dtype, std=1.0):
    t = torch.empty(shape, dtype=dtype, device="cuda")
    return t.normal_(0.0, std, generator=gen)


def _layer(case, gen, dtype):
    with torch.device("meta"):
        layer = MoELayer(case["d"], case["hidden"], case["experts"], case["top_k"])
    layer = layer.to(dtype).to_empty(device="cuda").requires_grad_(False)
    for p in layer.parameters():
        p.normal_(0.0, p.size(1) ** -0.5, generator=gen)
    return layer


def _segments(case):
    """Rows of every expert as uniform routing deals them; the same for every seed, since they are shapes."""
    rng = random.Random(case["tokens"] * 1009 + case["experts"])
    counts = [0] * case["experts"]
    for _ in range(case["tokens"]):
        for e in rng.sample(range(case["experts"]), case["top_k"]):
            counts[e] += 1
    return counts


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], _DTYPES[case["dtype"]]
    t, e, k = case["tokens"], case["experts"], case["top_k"]
    s = dict(kind=kind, top_k=k)
    if kind == "sinkhorn":
        s["router"] = SinkhornRouter(iters=10)
        s["logits"] = _randn(gen, (t, e), dtype)
        return s
    d = case["d"]
    x = _randn(gen, (t, d), dtype)
    if kind == "select_pack":
        return dict(s, x=x, logits=_randn(gen, (t, e), dtype))
    if kind == "layer":
        return dict(s, x=x.view(1, t, d), layer=_layer(case, gen, dtype))
    w_router = _randn(gen, (e, d), dtype, d ** -0.5)
    if kind == "route":
        s["skew"] = dict(skew_experts=min(8, e), skew_bias=2.0) if case["skew"] else {}
        return dict(s, x=x, w_router=w_router)
    h = case["hidden"]
    if kind == "grouped":
        # what a caller of the operator holds: the packed rows as one view per expert, the weights likewise
        weights = _randn(gen, (e, d, h), dtype, d ** -0.5)
        return dict(s, inputs=list(torch.split(x.repeat(k, 1), _segments(case))), weights=list(weights.unbind(0)))
    return dict(s, x=x, w_router=w_router, w1=_randn(gen, (e, h, d), dtype, d ** -0.5),
                w2=_randn(gen, (e, d, h), dtype, h ** -0.5))


@torch.no_grad()
def run(s):
    kind, k = s["kind"], s["top_k"]
    if kind == "route":
        o = ops.route_fused(s["x"], s["w_router"], k, **s["skew"])
        return {n: o[n] for n in _ROUTE_OUTPUTS}
    if kind == "select_pack":
        return fused_select_cuda.fused_select_forward(s["logits"], s["x"])
    if kind == "sinkhorn":
        return s["router"](s["logits"], k)
    if kind == "layer":
        return s["layer"](s["x"])
    if kind == "ffn":
        r = strategies.route("fused_select", s["x"], s["w_router"], k)
        return strategies.moe_forward(r, s["w1"], s["w2"], k)
    if kind == "grouped":
        return grouped_ffn_cuda.grouped_ffn_forward(s["inputs"], s["weights"])
    r = strategies.route("masked_matmul", s["x"], s["w_router"], k)
    return strategies.masked_matmul_forward(s["x"], r, s["w1"], s["w2"], k)


def _touched(case):
    """Experts that at least one token is routed to, as uniform routing deals them on average."""
    e, k = case["experts"], case["top_k"]
    return e * (1.0 - (1.0 - k / e) ** case["tokens"])


def work(case):
    kind, t, e, k = case["kind"], case["tokens"], case["experts"], case["top_k"]
    routing = t * k * 8  # picks and gates
    if kind == "sinkhorn":  # 16-bit logits in, int64 picks and 16-bit weights out; 10 row and column passes
        return dict(bytes=t * e * 2 + t * k * 10, flops=4.0 * 10 * t * e)
    d = case["d"]
    maps = e * 8
    if kind == "select_pack":
        return dict(bytes=t * e * 2 + routing + maps + (1 + k) * t * d * 2, flops=0.0)
    router = 2.0 * t * d * e
    if kind == "route":  # tokens and router weight in; routing, both maps and the packed rows out
        return dict(bytes=e * d * 2 + routing + 8 * t * k + maps + (1 + k) * t * d * 2, flops=router)
    h = case["hidden"]
    rows = t * k
    if kind == "grouped":
        return dict(bytes=rows * (d + h) * 2 + _touched(case) * d * h * 2, flops=2.0 * rows * d * h)
    if kind == "masked":
        return dict(bytes=2 * t * d * 2 + e * d * 2 + 2 * e * d * h * 2, flops=4.0 * t * e * d * h + router)
    mats = 3 if kind == "layer" else 2  # SwiGLU has a gate and an up matrix
    return dict(bytes=2 * t * d * 2 + e * d * 2 + _touched(case) * mats * d * h * 2, flops=2.0 * mats * rows * d * h + router)


def tolerance(case):
    kind, fp16 = case["kind"], case["dtype"] == "fp16"
    if kind in ("route", "select_pack"):
        # whole numbers and packed rows are the same; gates are fp32
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    # four times the distance to the same path in 64 bits
    if kind == "sinkhorn":  # 2.1e-4 / 1.7e-3: the weights are rounded to 16 bits; a pick may tie within fp32 rounding
        return {"rel": 9e-4 if fp16 else 7e-3, "max": 0.05, "differ": 1e-3}
    # 3.6e-4 / 2.9e-3 (largest 1.9e-3 / 1.5e-2): the hidden rows and the results are rounded to 16 bits
    return {"rel": 1.5e-3, "max": 8e-3} if fp16 else {"rel": 1.2e-2, "max": 6e-2}
