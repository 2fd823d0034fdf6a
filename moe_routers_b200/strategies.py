"""The four routing strategies of the reference's router benchmark (bench_router.py:434-438,
:468) as functions over the CUDA kernels: naive_topk, masked_matmul (A), fused_select (B),
sinkhorn (C).  Each returns the routing of a batch; `moe_forward` / `masked_matmul_forward` run
the expert FFNs on it (2-layer GELU FFN, weights [E, h, d] and [E, d, h])."""
from __future__ import annotations

import torch

from . import ops

STRATEGIES = ["naive_topk", "masked_matmul", "fused_select", "sinkhorn"]


def route(strategy: str, x: torch.Tensor, w_router: torch.Tensor, top_k: int, *, skew_experts: int = 0,
          skew_bias: float = 0.0, sinkhorn_iters: int = 10, sinkhorn_temperature: float = 1.0):
    """Routing of `x` under `strategy`.  Returns a dict with idx / gates and, for the strategies that
    permute (all but masked_matmul), counts / offsets / packed / row_route / route_row."""
    e = w_router.size(0)
    if strategy not in STRATEGIES:
        raise ValueError(f"Unknown strategies: {[strategy]}. Valid: {STRATEGIES}")
    if strategy == "fused_select":
        return ops.route_fused(x, w_router, top_k, skew_experts=skew_experts, skew_bias=skew_bias)
    if strategy == "naive_topk":
        # the same selection as fused_select (top-k of the logits, lowest index wins ties) with the
        # logits written out as well, as torch.topk on materialised logits would need them
        return ops.route_fused(x, w_router, top_k, skew_experts=skew_experts, skew_bias=skew_bias, return_logits=True)
    idx, gates, logits = ops.router_gemm_select(x, w_router, top_k, skew_experts=skew_experts,
                                                skew_bias=skew_bias, return_logits=True)
    if strategy == "sinkhorn":
        idx, gates = ops.sinkhorn(logits, top_k, iters=sinkhorn_iters, temperature=sinkhorn_temperature)
    out = dict(idx=idx, gates=gates, logits=logits)
    if strategy == "masked_matmul":
        return out  # Strategy A: no permutation
    counts, offsets, packed, row_route, route_row = ops.pack(x, idx, e)
    out.update(counts=counts, offsets=offsets, packed=packed, row_route=row_route, route_row=route_row)
    return out


def moe_forward(r: dict, w1: torch.Tensor, w2: torch.Tensor, top_k: int, activation: str = "gelu") -> torch.Tensor:
    """Sparse layer output from a routing with a packed buffer: grouped FFN + gate-weighted combine."""
    return ops.expert_ffn(r["packed"], w1, w2, r["offsets"], r["gates"], r["route_row"], top_k, activation=activation)


def masked_matmul_forward(x: torch.Tensor, r: dict, w1: torch.Tensor, w2: torch.Tensor, top_k: int,
                          activation: str = "gelu") -> torch.Tensor:
    """Strategy A: every expert runs densely over ALL tokens; outputs are summed with the top-k gate
    as mask (zero for unselected experts).  No permutation; E times the FLOPs of the sparse layer.
    Limited to 8 experts (the combine kernel sums at most 8 rows per token)."""
    t, d = x.shape
    e = w1.size(0)
    if e > 8:
        raise RuntimeError("masked_matmul_forward supports at most 8 experts")
    # All experts in one pair of launches, or as many at a time as keep the hidden rows within the bound.  One pair per
    # expert filled its last round of units each time, and the mask took four launches: 8 experts x 281 tokens,
    # 1792 -> 1152: 283 -> 59 us; 4 x 1389, 2368 -> 7264: 455 -> 388; 8 x 4096, 4096 -> 8192: 3865 -> 3755.
    at_once = max(1, _HIDDEN_BYTES // max(1, t * w1.size(1) * x.element_size()))
    if at_once >= e:  # (without slices, which take the host longer than the checks of what they give)
        y = ops.dense_experts(ops.dense_experts(x, w1, t, activation=activation), w2, t)
    else:
        y = torch.empty((e * t, d), dtype=x.dtype, device=x.device)
        for e0 in range(0, e, at_once):
            e1 = min(e, e0 + at_once)
            h = ops.dense_experts(x, w1[e0:e1], t, activation=activation)
            ops.dense_experts(h, w2[e0:e1], t, out=y[e0 * t:e1 * t])
    idx, gates = r["idx"], r["gates"]
    if not (idx.dim() == 2 and idx.shape == gates.shape and idx.size(0) == t and 1 <= idx.size(1) <= 8
            and idx.device == gates.device == x.device):
        # a routing of fewer tokens (the others get nothing), gates wider than the picks, more picks than the kernel takes:
        # as a mask over all experts, which raises where the shapes or devices do not go together
        mask = torch.zeros((t, e), dtype=torch.float32, device=x.device).scatter_add_(1, idx.long(), gates)
        idx, gates = torch.arange(e, dtype=torch.int32, device=x.device).expand(t, e), mask
    return ops.combine_dense(y, idx, gates, e)


_HIDDEN_BYTES = 512 << 20  # of masked_matmul_forward's hidden rows
