"""Strategy A's host side: what routings it takes, and what its operators refuse before they launch anything."""
import pytest
import torch


@pytest.fixture
def ops(monkeypatch):
    """CPU tensors get as far as the checks; there is nothing to launch on."""
    from moe_routers_b200 import build

    build.build_library()
    from moe_routers_b200 import ops

    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)
    return ops


@pytest.fixture
def masked_matmul(monkeypatch, ops):
    """The layer with its two operators as plain torch, with the shapes that the kernels index by."""
    def dense_experts(a, w, tokens, *, activation=None, out=None):
        e = w.size(0)
        assert a.size(0) in (tokens, e * tokens)
        rows = a.repeat(e, 1) if a.size(0) == tokens else a
        y = torch.bmm(rows.view(e, tokens, -1), w.transpose(1, 2)).view(e * tokens, -1)
        return y if out is None else out.copy_(y)

    def combine_dense(y, idx, gates, experts):
        t, picks = y.size(0) // experts, idx.size(1)
        assert idx.shape == gates.shape == (t, picks) and picks <= 8
        assert idx.numel() == 0 or 0 <= int(idx.min()) <= int(idx.max()) < experts
        out = torch.zeros(t, y.size(1))
        for j in range(picks):
            out += gates[:, j:j + 1] * y.view(experts, t, -1)[idx[:, j].long(), torch.arange(t)]
        return out

    monkeypatch.setattr(ops, "dense_experts", dense_experts)
    monkeypatch.setattr(ops, "combine_dense", combine_dense)
    from moe_routers_b200 import strategies

    return strategies.masked_matmul_forward


def _layer(t, e, d=8, h=16):
    g = torch.Generator().manual_seed(t)
    return [torch.randn(*s, generator=g) for s in ((t, d), (e, h, d), (e, d, h))]


@pytest.mark.parametrize("t,e,idx_shape,gates_shape,dtype", [
    (9, 4, (9, 2), (9, 2), torch.int32), (9, 8, (9, 8), (9, 8), torch.int64),
    (9, 4, (5, 2), (5, 2), torch.int32),    # a routing of fewer tokens: the others get nothing
    (9, 4, (0, 2), (0, 2), torch.int32),
    (9, 4, (9, 2), (9, 3), torch.int32),    # gates wider, or longer, than the picks
    (9, 4, (9, 2), (12, 2), torch.int32),
    (9, 3, (9, 12), (9, 12), torch.int64),  # more picks than the kernel takes
])
def test_routings_that_the_dense_layer_takes(masked_matmul, t, e, idx_shape, gates_shape, dtype):
    x, w1, w2 = _layer(t, e)
    g = torch.Generator().manual_seed(e)
    idx = torch.randint(0, e, idx_shape, generator=g).to(dtype)
    gates = torch.rand(gates_shape, generator=g)
    mask = torch.zeros(t, e).scatter_add_(1, idx.long(), gates)
    y = torch.stack([x @ a.t() @ b.t() for a, b in zip(w1, w2)])
    out = masked_matmul(x, dict(idx=idx, gates=gates), w1, w2, 2, activation=None)
    torch.testing.assert_close(out, torch.einsum("te,etd->td", mask, y))


@pytest.mark.parametrize("idx_shape,gates_shape", [((12, 2), (12, 2)), ((9, 2), (9, 1)), ((9, 2), (5, 2)), ((18,), (18,))])
def test_routings_that_it_refuses(masked_matmul, idx_shape, gates_shape):
    x, w1, w2 = _layer(9, 4)
    with pytest.raises(RuntimeError):
        masked_matmul(x, dict(idx=torch.zeros(idx_shape, dtype=torch.int32), gates=torch.zeros(gates_shape)),
                                         w1, w2, 2, activation=None)


@pytest.mark.parametrize("rows,idx_shape,gates_shape", [
    (32, (7, 2), (7, 2)), (32, (9, 2), (9, 2)), (33, (8, 2), (8, 2)), (32, (8, 2), (8, 1)), (32, (8, 2), (7, 2)), (32, (16,), (16,))])
def test_combine_dense_refuses_shapes_that_do_not_belong_together(ops, rows, idx_shape, gates_shape):
    with pytest.raises(RuntimeError, match="combine_dense: expected"):
        ops.combine_dense(torch.zeros(rows, 8, dtype=torch.float16), torch.zeros(idx_shape, dtype=torch.int32),
                          torch.zeros(gates_shape), 4)


@pytest.mark.parametrize("out", [
    torch.empty(31, 24, dtype=torch.float16), torch.empty(32, 16, dtype=torch.float16), torch.empty(32, 32, dtype=torch.float16),
    torch.empty(32, 24, dtype=torch.bfloat16), torch.empty(32, 48, dtype=torch.float16)[:, ::2], torch.empty(768, dtype=torch.float16),
    torch.empty(32, 24, dtype=torch.float16, device="meta")])
def test_dense_experts_refuses_an_output_that_is_not_its_own(ops, out):
    a, w = torch.zeros(8, 16, dtype=torch.float16), torch.zeros(4, 24, 16, dtype=torch.float16)
    with pytest.raises(RuntimeError, match="out must be"):
        ops.dense_experts(a, w, 8, out=out)
