"""What the operators refuse before they launch anything: sizes that the kernels would index by and that do not belong together."""
import pytest
import torch

from moe_routers_b200 import ops


@pytest.fixture(autouse=True)
def no_gpu(monkeypatch):
    """CPU tensors get as far as the checks; there is nothing to launch on."""
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)


def _half(*shape):
    return torch.zeros(*shape, dtype=torch.float16)


@pytest.mark.parametrize("route", [ops.route_fused, ops.router_gemm_select])
@pytest.mark.parametrize("w", [_half(8, 56), _half(8, 72), _half(8), _half(1, 8, 64)])
def test_router_weight_of_another_width(route, w):
    with pytest.raises(RuntimeError, match="router weight must be"):
        route(_half(4, 64), w, 2)


@pytest.mark.parametrize("logits", [_half(3, 8), _half(4, 7), _half(4, 16), _half(31), _half(2, 1, 8)])
def test_logits_of_another_shape(logits):
    with pytest.raises(RuntimeError, match="logits must be"):
        ops.fused_select(logits, _half(4, 64), 8, 2)
