"""The Sinkhorn kernel that keeps the matrix in registers, at the edges of its layouts: columns per lane,
rows per lane, CTAs per cluster, and the two kernels behind it (shared memory of one cluster; a cooperative grid), against the reference's iteration
(models/decoder_moe.py:92-123) in 64 bits."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [
    # tokens, experts, top_k, iters, dtype
    (1, 1, 1, 1, torch.float32), (1, 8, 8, 2, torch.float32), (512, 8, 1, 10, torch.float16),
    (513, 7, 2, 10, torch.float32), (65536, 8, 2, 3, torch.float16), (65537, 8, 2, 3, torch.float16),
    (257, 9, 4, 10, torch.bfloat16), (4097, 16, 4, 10, torch.float16), (2049, 17, 2, 10, torch.float32),
    (127, 32, 8, 4, torch.float32), (16384, 32, 2, 10, torch.bfloat16), (64, 33, 2, 10, torch.float32),
    (65, 60, 2, 10, torch.float16), (1025, 60, 4, 10, torch.float32), (2048, 64, 2, 10, torch.float32),
    (4096, 64, 8, 10, torch.float32), (8192, 64, 2, 10, torch.float32), (8193, 64, 2, 10, torch.float32),
    (33, 65, 2, 10, torch.float32), (4096, 128, 4, 10, torch.float32), (4097, 128, 4, 3, torch.float32),
    (17, 129, 2, 10, torch.float32), (2048, 256, 8, 10, torch.float16), (2049, 255, 2, 3, torch.float32),
    # a cooperative grid: one CTA, two, and as many as a large matrix takes (16384 x 64: 128 CTAs)
    (100, 257, 2, 10, torch.float32), (200, 257, 4, 10, torch.float32), (16384, 64, 2, 10, torch.float16),
    (16387, 128, 4, 10, torch.bfloat16),
]


def _exact(logits, k, iters, eps=1e-6):
    s = logits.double()
    q = torch.exp(s - s.max(dim=1, keepdim=True).values)
    for _ in range(iters):
        q = q / (q.sum(dim=1, keepdim=True) + eps)
        q = q / (q.sum(dim=0, keepdim=True) + eps) * (s.size(0) / s.size(1))
    q = q / (q.sum(dim=1, keepdim=True) + eps)
    vals, idx = torch.sort(q, dim=1, descending=True, stable=True)
    nxt = vals[:, k] if k < s.size(1) else torch.zeros_like(vals[:, 0]) - 1
    gaps = torch.cat([vals[:, :k], nxt[:, None]], dim=1)
    clear = ((gaps[:, :-1] - gaps[:, 1:]) > 1e-4 * vals[:, :1]).all(dim=1)  # not decided by fp32 rounding
    return idx[:, :k], vals[:, :k] / (vals[:, :k].sum(dim=1, keepdim=True) + eps), clear


@pytest.mark.parametrize("t,e,k,iters,dtype", CASES)
def test_sinkhorn_layout_edges(t, e, k, iters, dtype):
    from moe_routers_b200 import ops
    from moe_routers_b200.routers import SinkhornRouter

    g = torch.Generator().manual_seed(t * 7 + e)
    logits = torch.randn(t, e, generator=g).to(dtype).cuda()
    idx, w = ops.sinkhorn(logits, k, iters=iters)
    assert ops.read_status() == 0
    ref_idx, ref_w, clear = _exact(logits, k, iters)
    assert torch.equal(idx.long()[clear], ref_idx[clear])
    # 2 * iters + 1 normalisations, each a sum (a few ulp), a product and a division in fp32
    tol = (2 * iters + 1) * 16 * 2.0 ** -24
    torch.testing.assert_close(w.double()[clear], ref_w[clear], rtol=tol, atol=tol)
    # a second call on the same workspace, and the router's own result types: these values, rounded once
    ridx, rw = SinkhornRouter(iters=iters)(logits, k)
    assert ridx.dtype == torch.int64 and rw.dtype == dtype
    assert torch.equal(ridx, idx.long()) and torch.equal(rw, w.to(dtype))


@pytest.mark.parametrize("t,e", [(300, 64), (70, 16), (40, 256), (300, 60), (200, 257), (8193, 64), (16384, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_sinkhorn_masked_columns(t, e, dtype):
    """Logits of -inf or the type's lowest value are never picked while another is left, and weigh nothing, also
    where a whole column is masked (an expert that is switched off)."""
    from moe_routers_b200 import ops

    g = torch.Generator().manual_seed(t + e)
    for low in (float("-inf"), torch.finfo(dtype).min):
        a = torch.randn(t, e, generator=g).to(dtype)
        a[:, 3] = low
        a[:, e // 2:].masked_fill_(torch.rand(t, e - e // 2, generator=g) < 0.7, low)
        a = a.cuda()
        idx, w = ops.sinkhorn(a, 2)
        ref_idx, ref_w, clear = _exact(a, 2, 10)
        assert not (idx == 3).any() and torch.equal(idx.long()[clear], ref_idx[clear])
        tol = 21 * 16 * 2.0 ** -24  # as above
        torch.testing.assert_close(w.double()[clear], ref_w[clear], rtol=tol, atol=tol)
    assert ops.read_status() == 0


@pytest.mark.parametrize("t,e", [(300, 64), (70, 16), (40, 256), (300, 60), (200, 257), (8193, 64), (16384, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_sinkhorn_nan(t, e, dtype):
    """A NaN, a +inf or a row of -inf makes every sum NaN, as in the reference's arithmetic: all weights are NaN, and
    the picks stay column numbers."""
    from moe_routers_b200 import ops

    for bad in (lambda a: a[5].fill_(float("-inf")), lambda a: a[5, 3:4].fill_(float("inf")),
                lambda a: a[5, 3:4].fill_(float("nan"))):
        a = torch.randn(t, e, generator=torch.Generator().manual_seed(t + e)).to(dtype).cuda()
        bad(a)
        idx, w = ops.sinkhorn(a, 2)
        assert _exact(a, 2, 10)[1].isnan().all() and w.isnan().all()
        assert ((idx >= 0) & (idx < e)).all()
    assert ops.read_status() == 0


def test_sinkhorn_unaligned_logits():
    from moe_routers_b200 import ops

    g = torch.Generator().manual_seed(5)
    flat = torch.randn(300 * 64 + 1, generator=g).half().cuda()
    a = flat[1:].view(300, 64)  # rows 2 bytes off a 16-byte boundary
    b = a.clone()
    for x, y in zip(ops.sinkhorn(a, 4), ops.sinkhorn(b, 4)):
        assert torch.equal(x, y)


def _ctas(t, e):
    """CTAs of the one kernel that a call launches, read from its captured graph."""
    from cuda.bindings import driver

    from moe_routers_b200 import ops

    logits = torch.zeros(t, e, device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ops.sinkhorn(logits, 1)  # the stream's workspace exists
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        ops.sinkhorn(logits, 1)
    handle = driver.CUgraph(graph.raw_cuda_graph())
    _, _, count = driver.cuGraphGetNodes(handle)
    _, nodes, _ = driver.cuGraphGetNodes(handle, count)
    kernels = [n for n in nodes if driver.cuGraphNodeGetType(n)[1] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]
    assert len(kernels) == 1
    err, params = driver.cuGraphKernelNodeGetParams(kernels[0])
    assert err == driver.CUresult.CUDA_SUCCESS
    return params.gridDimX


def test_sinkhorn_keeps_the_portable_cluster_size_when_told():
    """MOE_B200_SINKHORN_CLUSTER=8, read once per process: every shape of this file in a process that has it
    set, and no cluster above 8 CTAs (4096 x 64 and 1024 x 256 fill 8 CTAs' registers)."""
    env = dict(os.environ, MOE_B200_SINKHORN_CLUSTER="8")
    here = os.path.abspath(__file__)
    root = os.path.dirname(os.path.dirname(here))
    code = (f"import sys; sys.path[:0] = [{root!r}, {os.path.dirname(here)!r}]; import test_sinkhorn_regs_gpu as t; "
            "print([t._ctas(*s) for s in ((4096, 64), (1024, 256), (600, 64))])")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, cwd=root)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip().endswith("[8, 8, 8]"), r.stdout
    r = subprocess.run([sys.executable, "-m", "pytest", here, "-q", "-x", "-k", "layout_edges or unaligned",
                        "-p", "no:cacheprovider"], env=env, capture_output=True, text=True, cwd=root)
    assert r.returncode == 0, r.stdout[-3000:]
