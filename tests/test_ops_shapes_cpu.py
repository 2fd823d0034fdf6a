"""What the operators refuse before they launch anything: sizes that the kernels would index by and that do not belong together."""
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


def _half(*shape):
    return torch.zeros(*shape, dtype=torch.float16)


@pytest.mark.parametrize("route", ["route_fused", "router_gemm_select"])
@pytest.mark.parametrize("w", [_half(8, 56), _half(8, 72), _half(8), _half(1, 8, 64)])
def test_router_weight_of_another_width(ops, route, w):
    with pytest.raises(RuntimeError, match="router weight must be"):
        getattr(ops, route)(_half(4, 64), w, 2)


@pytest.mark.parametrize("logits", [_half(3, 8), _half(4, 7), _half(4, 16), _half(31), _half(2, 1, 8)])
def test_logits_of_another_shape(ops, logits):
    with pytest.raises(RuntimeError, match="logits must be"):
        ops.fused_select(logits, _half(4, 64), 8, 2)


def _int32(*shape):
    return torch.zeros(*shape, dtype=torch.int32)


def test_offsets_of_fewer_experts(ops):
    with pytest.raises(RuntimeError, match="offsets must have"):
        ops.grouped_gemm(_half(6, 16), _half(4, 32, 16), _int32(4))
    with pytest.raises(RuntimeError, match="offsets must have"):
        ops.expert_ffn(_half(6, 16), _half(4, 32, 16), _half(4, 16, 32), _int32(4), torch.zeros(3, 2), _int32(6), 2, activation=None)


@pytest.mark.parametrize("gates,route_row", [((2, 2), 6), ((3, 1), 6), ((3, 3), 6), ((5,), 6), ((3, 2), 5)])
def test_maps_of_another_routing(ops, gates, route_row):
    with pytest.raises(RuntimeError, match="combine: "):
        ops.combine(_half(6, 16), torch.zeros(*gates), _int32(route_row), 2)
