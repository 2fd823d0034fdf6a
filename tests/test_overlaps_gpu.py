"""Kernels that set themselves up, or begin to copy, under the kernel in front of them: the same bits as one kernel after
another, at sizes where what starts early has to wait in the middle of its work."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _randn(*shape, dtype=torch.float16, seed=0, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _same(a, b):
    assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize("t,d,dtype", [(4096, 4096, torch.float16), (8192, 2048, torch.bfloat16)])
def test_select_behind_what_writes_its_inputs(t, d, dtype):
    """The rows are large enough for the early select.  Logits and rows are written right in front of every call."""
    from moe_routers_b200 import ops

    e, k, n = 64, 2, 5
    logits, rows = [_randn(t, e, dtype=dtype, seed=i) for i in range(n)], [_randn(t, d, dtype=dtype, seed=10 + i) for i in range(n)]
    now, x = torch.zeros_like(logits[0]), torch.zeros_like(rows[0])
    got = []
    for i in range(n):
        x.copy_(rows[i])
        now.copy_(logits[i])
        got.append(ops.fused_select(now, x, e, k))
    got += [ops.fused_select(logits[i], rows[i], e, k) for i in range(n)]  # and one behind the other's scatter
    assert ops.read_status() == 0
    for i, (idx, gates, counts, offsets, packed, row_route, route_row) in enumerate(got):
        want_idx, want_gates = ops.topk_select(logits[i % n], k)
        torch.cuda.synchronize()
        for a, b in zip((idx, gates, counts, offsets, packed, row_route, route_row),
                        (want_idx, want_gates, *ops.pack(rows[i % n], want_idx, e))):
            _same(a, b)


@pytest.mark.parametrize("counts,d,h,act,dtype", [
    # 320 to 480 units of the second GEMM for 74 pairs of CTAs, of 8 to 20 K stages; the first GEMM's last round is partial
    ([37] * 16, 5120, 2048, "gelu", torch.float16),
    ([1, 70, 0, 33] * 8, 5120, 2048, None, torch.bfloat16),
    ([16] * 8, 12288, 1024, "swiglu", torch.float16),
    ([3] * 60, 2048, 2304, "gelu", torch.bfloat16),
    ([300] * 4, 12288, 2560, "silu", torch.float16),
])
def test_second_gemm_with_early_weights(counts, d, h, act, dtype):
    """More units per pair of CTAs than are listed ahead and more stages than the ring has: the list and the weights that
    come early have to wait, for the first GEMM and then for their slots."""
    from moe_routers_b200 import ops

    e, rows = len(counts), sum(counts)
    ends = torch.tensor([0] + counts).cumsum(0).int().cuda()
    a = _randn(rows, d, dtype=dtype)
    w1 = _randn(e, 2 * h if act == "swiglu" else h, d, dtype=dtype, seed=1, std=d ** -0.5)
    w2 = _randn(e, d, h, dtype=dtype, seed=2, std=h ** -0.5)
    gates = torch.rand(rows, 1, device="cuda")
    back = torch.randperm(rows, device="cuda").int()
    want = ops.grouped_gemm(a, w1, ends, activation=act)
    torch.cuda.synchronize()
    want = ops.grouped_gemm(want, w2, ends)
    torch.cuda.synchronize()
    want = ops.combine(want, gates, back, 1)
    for _ in range(3):
        _same(ops.expert_ffn(a, w1, w2, ends, gates, back, 1, activation=act), want)
    assert ops.read_status() == 0


@pytest.mark.parametrize("tokens,d,h,e,k", [(16, 576, 1088, 16, 2), (33, 1024, 256, 64, 4), (3330, 768, 512, 32, 2)])
def test_layers_behind_one_another(tokens, d, h, e, k):
    """A layer's router starts under the combine that writes its tokens."""
    from moe_routers_b200 import ops
    from moe_routers_b200._lib import lib
    from moe_routers_b200.moe_layer import MoELayer

    torch.manual_seed(tokens)
    layers = [MoELayer(d, h, e, k).half().cuda().requires_grad_(False) for _ in range(4)]
    x = _randn(1, tokens, d, seed=tokens)
    y = x
    for layer in layers:  # outputs as large as inputs, so that the last layer still routes on something
        scale = 1.0 / float(layer(y).float().std())
        for expert in layer.experts:
            expert.w2.weight.mul_(scale)
        y = layer(y)

    def chain(x):
        outs = []
        for layer in layers:
            x = layer(x)
            outs.append(x)
        return outs

    lib.moe_set_pdl(0)
    try:
        want = chain(x)
        torch.cuda.synchronize()
    finally:
        lib.moe_set_pdl(1)
    assert all(torch.isfinite(y).all() and 0.5 < y.float().std() < 2 for y in want)
    for _ in range(3):
        for a, b in zip(chain(x), want):
            _same(a, b)
    assert ops.read_status() == 0


def test_a_captured_select_is_launched_plainly():
    """Among the kernels of a graph an early start of the select costs time: only the scatters start under their selects."""
    from moe_routers_b200 import ops

    x, logits = _randn(4096, 4096), _randn(4096, 64, seed=1)
    want = ops.fused_select(logits, x, 64, 2)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        got = [ops.fused_select(logits, x, 64, 2) for _ in range(3)]
    driver, count = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(16)
    nodes, edges = [(ctypes.c_void_p * 16)() for _ in range(2)], (ctypes.c_ubyte * 8 * 16)()  # from_port, to_port, type, ..
    assert driver.cuGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), *nodes, edges, ctypes.byref(count)) == 0
    assert [e[2] for e in edges[:count.value]].count(1) == 3  # 1: CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC
    graph.instantiate()
    graph.replay()
    for outs in got:
        for a, b in zip(outs, want):
            _same(a, b)
