"""Torch-facing operators over the C ABI of libmoe_b200.so.

PyTorch is used for device memory and streams only: every function allocates
its outputs with torch, passes raw device pointers and the current stream to
the library and returns torch tensors.  All compute happens in the CUDA
kernels of the library; there is no CPU or eager fallback, CPU tensors are
rejected.
"""
from __future__ import annotations

import contextlib
import ctypes
from typing import Optional

import torch

from . import _host, _lib
from ._host import empties
from ._lib import check, lib

_DTYPE_CODE = {torch.float16: _lib.MOE_F16, torch.bfloat16: _lib.MOE_BF16, torch.float32: _lib.MOE_F32}

_MAX_ROWS = 2 ** 31 - 1  # what the library's int arguments hold

_workspaces: dict = {}


# The current stream's handle and the current device, without building a Stream or Device object.
_raw_stream = torch._C._cuda_getCurrentRawStream
_current_device = torch._C._cuda_getDevice
_SAME_DEVICE = contextlib.nullcontext()


def _stream() -> int:
    return _raw_stream(_current_device())


def _on(index: int):
    """Makes CUDA device `index` current for a `with` block (nothing to do where it is)."""
    return _SAME_DEVICE if index == _current_device() else torch.cuda.device(index)


def _require_cuda(*tensors: torch.Tensor) -> None:
    for t in tensors:
        if not t.is_cuda:
            raise RuntimeError("inputs must be CUDA")  # same text as kernels/fused_select.cu:205


def workspace(device: torch.device, tokens: int, experts: int, top_k: int) -> torch.Tensor:
    """Per (device, stream) scratch buffer, grown on demand and initialised once."""
    return _workspace(device.index if device.index is not None else torch.cuda.current_device(), tokens, experts, top_k)


def _workspace(index: int, tokens: int, experts: int, top_k: int) -> torch.Tensor:
    need = max(lib.moe_workspace_bytes(int(tokens), int(experts), int(top_k)), 1 << 16)
    key = (index, _stream())
    ws = _workspaces.get(key)
    if ws is None or ws.numel() < need:
        ws = torch.empty(max(need, 1 << 20), dtype=torch.uint8, device=torch.device("cuda", index))
        check(lib.moe_workspace_init(ws.data_ptr(), ws.numel(), _stream()))
        _workspaces[key] = ws
    return ws


# The operators that _host runs as one native call where their arguments are plain; the functions below take the rest.
_host.bind({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value
            for name in ("moe_workspace_bytes", "moe_route_fused", "moe_fused_select", "moe_sinkhorn", "moe_sinkhorn_router",
                         "moe_grouped_gemm", "moe_expert_ffn", "moe_store_offsets")}, _workspaces, _workspace, check)


def read_status(device: Optional[torch.device] = None) -> int:
    """Synchronise the current stream and raise if a kernel recorded an error."""
    device = device or torch.device("cuda", torch.cuda.current_device())
    ws = workspace(device, 1, 1, 1)
    out = ctypes.c_int(0)
    check(lib.moe_read_status(ws.data_ptr(), _stream(), ctypes.byref(out)))
    return out.value


def topk_select(logits: torch.Tensor, top_k: int):
    """(idx int32 [T,k], gates float32 [T,k]): lowest index wins ties."""
    _require_cuda(logits)
    if logits.dim() != 2:
        raise RuntimeError("logits shape must be [T, E]")
    if logits.dtype not in _DTYPE_CODE:
        raise RuntimeError("logits must be fp16/bf16/fp32")
    logits = logits.contiguous()
    t, e = logits.shape
    dev = logits.get_device()
    with _on(dev):
        idx, gates = empties(dev, ((torch.int32, t, top_k), (torch.float32, t, top_k)))
        check(lib.moe_topk_select(logits.data_ptr(), _DTYPE_CODE[logits.dtype], t, e, int(top_k),
                                  idx.data_ptr(), gates.data_ptr(), _stream()))
    return idx, gates


def _map_specs(t: int, experts: int, k: int):
    """counts, offsets, row_route, route_row"""
    return (torch.int32, experts), (torch.int32, experts + 1), (torch.int32, t * k), (torch.int32, t * k)


def _route_specs(t: int, d: int, experts: int, k: int, dtype: torch.dtype):
    """idx, gates, packed, counts, offsets, row_route, route_row"""
    return ((torch.int32, t, k), (torch.float32, t, k), (dtype, t * k, d)) + _map_specs(t, experts, k)


def pack(x: torch.Tensor, idx: torch.Tensor, experts: int, *, copy_rows: bool = True):
    """Expert-contiguous pack.  Returns (counts, offsets, packed, row_route, route_row)."""
    _require_cuda(x, idx)
    if x.dim() != 2 or idx.dim() != 2 or idx.size(0) != x.size(0):
        raise RuntimeError("x shape must be [T, d_model] and idx [T, k]")
    if x.element_size() not in (2, 4):
        raise RuntimeError("x must have 2- or 4-byte elements")
    x = x.contiguous()
    idx = idx.to(torch.int32).contiguous()
    t, d = x.shape
    k = idx.size(1)
    dev = x.get_device()
    with _on(dev):
        counts, offsets, row_route, route_row = empties(dev, _map_specs(t, experts, k))
        packed = empties(dev, ((x.dtype, t * k, d),))[0] if copy_rows else None
        ws = _workspace(dev, t, experts, k)
        check(lib.moe_pack(x.data_ptr(), x.element_size(), idx.data_ptr(), t, d, int(experts), k,
                           counts.data_ptr(), offsets.data_ptr(),
                           packed.data_ptr() if packed is not None else None,
                           row_route.data_ptr(), route_row.data_ptr(), ws.data_ptr(), ws.numel(),
                           _stream()))
    return counts, offsets, packed, row_route, route_row


def pack_scatter(x: torch.Tensor, experts: int, out: dict) -> dict:
    """Re-run only the scatter half of `route_fused` into the buffers of `out` (a dict returned by
    route_fused for the same x).  The per-tile histograms of that call are read from
    `out["workspace"]`, the scratch buffer route_fused used (scratch is per stream, so the buffer of
    the calling stream would be the wrong one after a stream switch); no other route may have run
    on that buffer in between."""
    _require_cuda(x)
    t, d = x.shape
    k = out["idx"].size(1)
    with _on(x.get_device()):
        ws = out["workspace"]
        check(lib.moe_pack_scatter(x.data_ptr(), x.element_size(), out["idx"].data_ptr(), t, d, int(experts), k,
                                   out["counts"].data_ptr(), out["offsets"].data_ptr(), out["packed"].data_ptr(),
                                   out["row_route"].data_ptr(), out["route_row"].data_ptr(), ws.data_ptr(),
                                   ws.numel(), _stream()))
    return out


def route_plan(x: torch.Tensor, idx: torch.Tensor, experts: int, *, hist_ready: bool = False) -> dict:
    """Counts, offsets and the route <-> row maps of a pack, without copying a row.

    `hist_ready`: the per-tile histograms of `idx` are already in the calling stream's scratch buffer
    (router_gemm_select has just produced idx on this stream); otherwise they are computed from idx.
    Returns dict(idx, counts, offsets, row_route, route_row, workspace) for `pack_scatter_to`."""
    _require_cuda(x, idx)
    idx = idx.to(torch.int32).contiguous()
    t, d = x.shape
    k = idx.size(1)
    dev = x.get_device()
    with _on(dev):
        counts, offsets, row_route, route_row = empties(dev, _map_specs(t, experts, k))
        ws = _workspace(dev, t, experts, k)
        o = dict(idx=idx, counts=counts, offsets=offsets, row_route=row_route, route_row=route_row, workspace=ws)
        fn = lib.moe_pack_scatter if hist_ready else lib.moe_pack
        check(fn(x.data_ptr(), x.element_size(), idx.data_ptr(), t, d, int(experts), k, o["counts"].data_ptr(),
                 o["offsets"].data_ptr(), None, o["row_route"].data_ptr(), o["route_row"].data_ptr(),
                 ws.data_ptr(), ws.numel(), _stream()))
    return o


def pack_scatter_to(x: torch.Tensor, experts: int, plan: dict, seg_base: torch.Tensor) -> dict:
    """Scatter the token rows of a planned route to one destination segment per expert: rows of expert
    e go, in canonical order, to the address seg_base[e] onwards (int64 [experts] on the device;
    16-byte aligned; peers' mapped memory allowed).  `plan` comes from `route_plan` (or route_fused)
    for the same x; its histograms must still be in plan["workspace"]."""
    _require_cuda(x, seg_base)
    if seg_base.dtype != torch.int64 or seg_base.numel() < experts:
        raise RuntimeError("seg_base must be an int64 tensor with one address per expert")
    x = x.contiguous()
    t, d = x.shape
    k = plan["idx"].size(1)
    ws = plan["workspace"]
    with _on(x.get_device()):
        check(lib.moe_pack_scatter_to(x.data_ptr(), x.element_size(), plan["idx"].data_ptr(), t, d, int(experts), k,
                                      plan["counts"].data_ptr(), plan["offsets"].data_ptr(), seg_base.data_ptr(),
                                      plan["row_route"].data_ptr(), plan["route_row"].data_ptr(), ws.data_ptr(),
                                      ws.numel(), _stream()))
    return plan


def fused_select(logits: torch.Tensor, x: torch.Tensor, experts: int, top_k: int, out: Optional[tuple] = None):
    """Select + count + scan + pack from given logits in two launches.
    Returns (idx, gates, counts, offsets, packed, row_route, route_row); `out` may be the tuple a
    previous call returned, to reuse its buffers."""
    if out is None and x.is_cuda:
        dev = _current_device()
        o = _host.fused_select(dev, _raw_stream(dev), logits, x, experts, top_k)
        if o is not None:
            return o
    _require_cuda(logits, x)
    if logits.dtype not in _DTYPE_CODE:
        raise RuntimeError("logits must be fp16/bf16/fp32")
    t, d = x.shape
    if logits.numel() < t * experts or (logits.numel() > t * experts and logits.dim() > 1 and logits.size(-1) != experts):
        raise RuntimeError("logits must be [T, n_experts] for x [T, d_model]")
    logits = logits.contiguous()
    x = x.contiguous()
    dev = x.get_device()
    with _on(dev):
        if out is None:
            idx, gates, packed, counts, offsets, row_route, route_row = empties(dev, _route_specs(t, d, experts, top_k, x.dtype))
            out = (idx, gates, counts, offsets, packed, row_route, route_row)
        else:
            idx, gates, counts, offsets, packed, row_route, route_row = out
        ws = _workspace(dev, t, experts, top_k)
        check(lib.moe_fused_select(logits.data_ptr(), _DTYPE_CODE[logits.dtype], x.data_ptr(), x.element_size(), t, d,
                                   int(experts), int(top_k), idx.data_ptr(), gates.data_ptr(), counts.data_ptr(),
                                   offsets.data_ptr(), packed.data_ptr(), row_route.data_ptr(), route_row.data_ptr(),
                                   ws.data_ptr(), ws.numel(), _stream()))
    return out


def combine(y: torch.Tensor, gates: torch.Tensor, route_row: torch.Tensor, top_k: int) -> torch.Tensor:
    """out[t] = sum_j gates[t,j] * y[route_row[t*k+j]]."""
    _require_cuda(y, gates, route_row)
    if y.dtype not in (torch.float16, torch.bfloat16):
        raise RuntimeError("y must be fp16 or bf16")
    y = y.contiguous()
    gates = gates.to(torch.float32).contiguous()
    route_row = route_row.to(torch.int32).contiguous()
    rows, d = y.shape
    t = rows // top_k
    if gates.numel() < t * top_k or (gates.numel() > t * top_k and gates.dim() > 1 and gates.size(-1) != top_k):
        raise RuntimeError("combine: gates must be [T, top_k] for y [T * top_k, d]")
    if route_row.numel() < t * top_k:
        raise RuntimeError("combine: route_row must have one row per route")
    dev = y.get_device()
    with _on(dev):
        out, = empties(dev, ((y.dtype, t, d),))
        check(lib.moe_combine(y.data_ptr(), _DTYPE_CODE[y.dtype], gates.data_ptr(), route_row.data_ptr(),
                              t, d, int(top_k), out.data_ptr(), _stream()))
    return out


def _check_router_weight(x: torch.Tensor, w_router: torch.Tensor) -> None:
    if w_router.dim() != 2 or x.dim() != 2 or w_router.size(1) != x.size(1):
        raise RuntimeError("x must be [T, d_model] and the router weight must be [n_experts, d_model]")


def router_gemm_select(x: torch.Tensor, w_router: torch.Tensor, top_k: int, *, skew_experts: int = 0,
                       skew_bias: float = 0.0, return_logits: bool = False):
    """Fused logit GEMM + skew + top-k + gates.  Returns (idx, gates[, logits fp32])."""
    _require_cuda(x, w_router)
    if x.dtype not in (torch.float16, torch.bfloat16) or w_router.dtype != x.dtype:
        raise RuntimeError("x and the router weight must both be fp16 (Half) or both bf16")
    _check_router_weight(x, w_router)
    x = x.contiguous()
    w_router = w_router.contiguous()
    t, d = x.shape
    e = w_router.size(0)
    dev = x.get_device()
    with _on(dev):
        idx, gates = empties(dev, ((torch.int32, t, top_k), (torch.float32, t, top_k)))
        logits = empties(dev, ((torch.float32, t, e),))[0] if return_logits else None
        ws = _workspace(dev, t, e, top_k)
        check(lib.moe_router_gemm_select(x.data_ptr(), w_router.data_ptr(), _DTYPE_CODE[x.dtype], t, d, e, int(top_k),
                                         int(skew_experts), float(skew_bias), idx.data_ptr(),
                                         gates.data_ptr(), logits.data_ptr() if return_logits else None,
                                         ws.data_ptr(), ws.numel(), _stream()))
    return (idx, gates, logits) if return_logits else (idx, gates)


def route_fused(x: torch.Tensor, w_router: torch.Tensor, top_k: int, *, skew_experts: int = 0,
                skew_bias: float = 0.0, return_logits: bool = False, out: Optional[dict] = None):
    """The whole fused_select strategy: logit GEMM + select + count/scan/pack.

    Returns a dict with idx, gates, counts, offsets, packed, row_route,
    route_row (and logits when asked), plus `workspace`: the scratch buffer
    of the calling stream, which holds the per-tile histograms of this call
    until the next route on that stream.  `out` may carry pre-allocated
    tensors from a previous call to avoid re-allocation.
    """
    if out is None and x.is_cuda:
        dev = _current_device()
        o = _host.route(dev, _raw_stream(dev), x, w_router, top_k, skew_experts, skew_bias, bool(return_logits))
        if o is not None:
            return o
    _require_cuda(x, w_router)
    if x.dtype not in (torch.float16, torch.bfloat16) or w_router.dtype != x.dtype:
        raise RuntimeError("x and the router weight must both be fp16 (Half) or both bf16")
    _check_router_weight(x, w_router)
    x = x.contiguous()
    w_router = w_router.contiguous()
    t, d = x.shape
    e = w_router.size(0)
    dev = x.get_device()
    with _on(dev):
        o = out if out is not None else {}
        if "idx" not in o:
            idx, gates, packed, counts, offsets, row_route, route_row = empties(dev, _route_specs(t, d, e, top_k, x.dtype))
            o.update(idx=idx, gates=gates, counts=counts, offsets=offsets, packed=packed, row_route=row_route,
                     route_row=route_row)
        if return_logits and "logits" not in o:
            o["logits"], = empties(dev, ((torch.float32, t, e),))
        ws = o["workspace"] = _workspace(dev, t, e, top_k)
        check(lib.moe_route_fused(x.data_ptr(), w_router.data_ptr(), _DTYPE_CODE[x.dtype], t, d, e, int(top_k),
                                  int(skew_experts), float(skew_bias), o["idx"].data_ptr(),
                                  o["gates"].data_ptr(), o["counts"].data_ptr(), o["offsets"].data_ptr(),
                                  o["packed"].data_ptr(), o["row_route"].data_ptr(),
                                  o["route_row"].data_ptr(),
                                  o["logits"].data_ptr() if return_logits else None,
                                  ws.data_ptr(), ws.numel(), _stream()))
    return o


def sinkhorn(logits: torch.Tensor, top_k: int, *, iters: int = 10, epsilon: float = 1e-6,
             temperature: float = 1.0):
    """Sinkhorn-balanced top-k: (idx int32 [T,k], gates float32 [T,k])."""
    return _sinkhorn(False, logits, top_k, iters, epsilon, temperature)


def sinkhorn_router(logits: torch.Tensor, top_k: int, *, iters: int = 10, epsilon: float = 1e-6,
                    temperature: float = 1.0):
    """The same as the router plug-in returns it: (idx int64 [T,k], weights [T,k] in the logits' type)."""
    return _sinkhorn(True, logits, top_k, iters, epsilon, temperature)


def _sinkhorn(router: bool, logits, top_k, iters, epsilon, temperature):
    if logits.is_cuda:
        dev = _current_device()
        o = _host.sinkhorn(dev, _raw_stream(dev), router, logits, top_k, iters, epsilon, temperature)
        if o is not None:
            return o
    _require_cuda(logits)
    entry, idx_dtype, gate_dtype = ((lib.moe_sinkhorn_router, torch.int64, logits.dtype) if router else
                                    (lib.moe_sinkhorn, torch.int32, torch.float32))
    if logits.dim() != 2:
        raise ValueError("SinkhornRouter expects logits of shape [tokens, experts]")
    if logits.dtype not in _DTYPE_CODE:
        raise RuntimeError("logits must be fp16/bf16/fp32")
    logits = logits.contiguous()
    t, e = logits.shape
    dev = logits.get_device()
    with _on(dev):
        idx, gates = empties(dev, ((idx_dtype, t, top_k), (gate_dtype, t, top_k)))
        ws = _workspace(dev, t, e, top_k)
        check(entry(logits.data_ptr(), _DTYPE_CODE[logits.dtype], t, e, int(top_k), int(iters), float(epsilon),
                    float(temperature), idx.data_ptr(), gates.data_ptr(), ws.data_ptr(), ws.numel(), _stream()))
    return idx, gates


_ACT = {None: _lib.MOE_ACT_NONE, "none": _lib.MOE_ACT_NONE, "gelu": _lib.MOE_ACT_GELU,
        "silu": _lib.MOE_ACT_SILU, "swiglu": _lib.MOE_ACT_SWIGLU}


def grouped_gemm(a: torch.Tensor, w: torch.Tensor, offsets: torch.Tensor, *, layout: str = "nk",
                 activation: Optional[str] = None, row_scale: Optional[torch.Tensor] = None,
                 out: Optional[torch.Tensor] = None, sm_margin: int = 0,
                 bias: Optional[torch.Tensor] = None, out_rows: Optional[torch.Tensor] = None) -> torch.Tensor:
    """c[offsets[e]:offsets[e+1]] = act(a[offsets[e]:offsets[e+1]] @ W[e]) for every expert.

    a [rows, K]; w [E, N, K] (layout "nk") or [E, K, N] (layout "kn"); both fp16 or both bf16;
    offsets int32 [E+1] on the device; bias [E, output features] (same dtype) is added before the
    activation.  With activation "swiglu" the weight has
    2N output features (gate rows first, then up) and the result has N columns.
    With `out_rows` (int64 [rows] on the device: one 16-byte aligned address per result row, possibly
    in a mapped peer buffer) the rows are stored there instead of in a dense result, and the table
    itself is returned.
    """
    _require_cuda(a, w, offsets)
    if a.dtype not in (torch.float16, torch.bfloat16) or w.dtype != a.dtype:
        raise RuntimeError("grouped_gemm: a and w must both be fp16 or both bf16")
    if bias is not None and (bias.dtype != a.dtype or not bias.is_cuda):
        raise RuntimeError("grouped_gemm: bias must be a CUDA tensor of the same dtype")
    if w.dim() != 3:
        raise RuntimeError("grouped_gemm: w must be [E, N, K] or [E, K, N]")
    a = a.contiguous()
    w = w.contiguous()
    offsets = offsets.to(torch.int32).contiguous()
    rows, k_dim = a.shape
    e = w.size(0)
    n_w = w.size(1) if layout == "nk" else w.size(2)
    if (w.size(2) if layout == "nk" else w.size(1)) != k_dim:
        raise RuntimeError("grouped_gemm: inner dimensions differ")
    if offsets.numel() <= e:
        raise RuntimeError("grouped_gemm: offsets must have experts + 1 entries")
    act = _ACT[activation]
    n_out = n_w // 2 if act == _lib.MOE_ACT_SWIGLU else n_w
    dev = a.get_device()
    with _on(dev):
        ws = _workspace(dev, 1, e, 1)
        rs = row_scale.to(torch.float32).contiguous() if row_scale is not None else None
        if out_rows is not None:
            if out_rows.dtype != torch.int64 or not out_rows.is_cuda or out_rows.numel() < rows:
                raise RuntimeError("grouped_gemm: out_rows must be a CUDA int64 tensor with one address per row")
            check(lib.moe_grouped_gemm_rows(a.data_ptr(), w.data_ptr(), out_rows.data_ptr(), offsets.data_ptr(), e,
                                            rows, k_dim, n_out,
                                            _lib.MOE_W_NK if layout == "nk" else _lib.MOE_W_KN, w.stride(0), act,
                                            rs.data_ptr() if rs is not None else None,
                                            bias.contiguous().data_ptr() if bias is not None else None,
                                            _DTYPE_CODE[a.dtype], int(sm_margin), ws.data_ptr(), ws.numel(),
                                            _stream()))
            return out_rows
        c = out if out is not None else empties(dev, ((a.dtype, rows, n_out),))[0]
        check(lib.moe_grouped_gemm(a.data_ptr(), w.data_ptr(), c.data_ptr(), offsets.data_ptr(), e, rows,
                                   k_dim, n_out, _lib.MOE_W_NK if layout == "nk" else _lib.MOE_W_KN,
                                   w.stride(0), act, rs.data_ptr() if rs is not None else None,
                                   bias.contiguous().data_ptr() if bias is not None else None,
                                   _DTYPE_CODE[a.dtype], int(sm_margin),
                                   ws.data_ptr(), ws.numel(), _stream()))
    return c


def dense_experts(a: torch.Tensor, w: torch.Tensor, tokens: int, *, activation: Optional[str] = None,
                  out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """c[e * tokens + t] = act(a[row] @ W[e].T) for every expert and token: row = t where `a` has `tokens` rows, which
    all experts read, else e * tokens + t.  w [E, N, K]; fp16 or bf16."""
    _require_cuda(a, w)
    if a.dtype not in (torch.float16, torch.bfloat16) or w.dtype != a.dtype:
        raise RuntimeError("grouped_gemm: a and w must both be fp16 or both bf16")
    if a.dim() != 2 or w.dim() != 3:
        raise RuntimeError("dense_experts: expected a [rows, K] and w [E, N, K]")
    a = a.contiguous()
    w = w.contiguous()
    e, n_w, k_dim = w.shape
    if a.size(1) != k_dim:
        raise RuntimeError("grouped_gemm: inner dimensions differ")
    if a.size(0) not in (tokens, e * tokens):
        raise RuntimeError("dense_experts: a must have tokens or experts * tokens rows")
    if e * tokens > _MAX_ROWS:
        raise RuntimeError("dense_experts: too many rows")
    act = _ACT[activation]
    n_out = n_w // 2 if act == _lib.MOE_ACT_SWIGLU else n_w
    if out is not None and (out.shape != (e * tokens, n_out) or out.dtype != a.dtype or out.device != a.device
                            or not out.is_contiguous()):
        raise RuntimeError(f"dense_experts: out must be a contiguous [{e * tokens}, {n_out}] tensor like a")
    dev = a.get_device()
    with _on(dev):
        ws = _workspace(dev, 1, e, 1)
        c = out if out is not None else empties(dev, ((a.dtype, e * tokens, n_out),))[0]
        check(lib.moe_dense_experts(a.data_ptr(), w.data_ptr(), c.data_ptr(), e, tokens, int(a.size(0) == tokens), k_dim, n_out,
                                    _lib.MOE_W_NK, w.stride(0), act, _DTYPE_CODE[a.dtype], ws.data_ptr(), ws.numel(),
                                    _stream()))
    return c


def combine_dense(y: torch.Tensor, idx: torch.Tensor, gates: torch.Tensor, experts: int) -> torch.Tensor:
    """out[t] = sum_e g[t, e] * y[e * T + t] with the gate of t's pick of expert e, 0 for the experts not picked.
    A pick outside [0, E) adds nothing and is reported by `read_status`."""
    _require_cuda(y, idx, gates)
    if y.dtype not in (torch.float16, torch.bfloat16):
        raise RuntimeError("y must be fp16 or bf16")
    if y.dim() != 2 or idx.dim() != 2 or idx.shape != gates.shape or y.size(0) != experts * idx.size(0):
        raise RuntimeError("combine_dense: expected y [experts * T, d] and idx, gates [T, top_k]")
    if y.size(0) > _MAX_ROWS:
        raise RuntimeError("combine_dense: too many rows")
    y = y.contiguous()
    idx = idx.to(torch.int32).contiguous()
    gates = gates.to(torch.float32).contiguous()
    t, d = idx.size(0), y.size(1)
    dev = y.get_device()
    with _on(dev):
        out, = empties(dev, ((y.dtype, t, d),))
        stream = _stream()
        ws = _workspaces.get((dev, stream))  # (of any size: only its status word is used)
        if ws is None:
            ws = _workspace(dev, 1, 1, 1)
        check(lib.moe_combine_dense_checked(y.data_ptr(), _DTYPE_CODE[y.dtype], idx.data_ptr(), gates.data_ptr(), t, d,
                                            int(experts), idx.size(1), out.data_ptr(), ws.data_ptr(), stream))
    return out


def expert_ffn(rows: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor, offsets: torch.Tensor, gates: torch.Tensor,
               route_row: torch.Tensor, top_k: int, *, activation: Optional[str]) -> torch.Tensor:
    """Two grouped GEMMs ([E, N, K] weights, the activation after the first) over the packed rows, then the
    gate-weighted combine."""
    if rows.is_cuda:
        dev = _current_device()
        o = _host.expert_ffn(dev, _raw_stream(dev), rows, w1, w2, offsets, _ACT[activation], gates, route_row, top_k)
        if o is not None:
            return o
    h = grouped_gemm(rows, w1, offsets, layout="nk", activation=activation)
    y = grouped_gemm(h, w2, offsets, layout="nk")
    return combine(y, gates, route_row, top_k)


def grouped_lists(inputs: list, weights: list) -> Optional[list]:
    """[M_i, K] inputs times [K, N] weights, pair by pair, where both lists are consecutive views of one fp16 buffer
    each; None, with nothing done, where they are not or a stream is being captured."""
    dev = _current_device()
    if torch.cuda.is_current_stream_capturing():
        return None  # (the general path uploads the offsets in a way that a capture refuses, as it always has)
    return _host.grouped_lists(dev, _raw_stream(dev), inputs, weights)
