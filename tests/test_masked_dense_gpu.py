"""Strategy A in one pair of launches: the same bits as one grouped GEMM per expert and a gate-masked fp32 sum, at token
counts around the column steps, with the hidden rows in one piece and in several."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _per_expert(x, idx, gates, w1, w2):
    from moe_routers_b200 import ops

    t = x.size(0)
    seg = torch.tensor([0, t], dtype=torch.int32, device="cuda")
    out = torch.zeros(t, w2.size(1), device="cuda")
    for e in range(w1.size(0)):
        h = ops.grouped_gemm(x, w1[e:e + 1], seg, activation="gelu")
        y = ops.grouped_gemm(h, w2[e:e + 1], seg).float()
        out = torch.addcmul(out, (gates * (idx == e)).sum(1, keepdim=True), y)
    return out


@pytest.mark.parametrize("t,d,h,e,k,dtype", [
    (1, 64, 64, 1, 1, torch.float16), (31, 64, 96, 3, 2, torch.bfloat16), (33, 528, 272, 8, 8, torch.float16),
    (257, 320, 512, 4, 2, torch.bfloat16), (1000, 144, 1040, 8, 2, torch.float16), (2400, 64, 64, 8, 1, torch.float16)])
@pytest.mark.parametrize("pieces", [1, 2])
def test_same_as_one_gemm_per_expert(t, d, h, e, k, dtype, pieces, monkeypatch):
    from moe_routers_b200 import ops, strategies

    if pieces > 1:
        monkeypatch.setattr(strategies, "_HIDDEN_BYTES", 2 * t * h * -(-e // pieces))
    g = torch.Generator(device="cuda").manual_seed(t)
    draw = lambda *s, std=1.0: torch.empty(*s, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)  # noqa: E731
    x, w1, w2 = draw(t, d), draw(e, h, d, std=d ** -0.5), draw(e, d, h, std=h ** -0.5)
    idx = torch.rand(t, e, device="cuda", generator=g).argsort(1)[:, :k].int()
    gates = torch.rand(t, k, device="cuda", generator=g)
    out = strategies.masked_matmul_forward(x, dict(idx=idx, gates=gates), w1, w2, k)
    assert ops.read_status() == 0
    # the same products and the same fp32 sums in the same order; one rounding to 16 bits (fused or not: one ulp)
    ulp = 2.0 ** (-10 if dtype == torch.float16 else -7)
    torch.testing.assert_close(out.float(), _per_expert(x, idx, gates, w1, w2), rtol=ulp, atol=1e-6)


def test_infinite_rows_of_experts_not_picked_still_count():
    """0 * inf is NaN, as where the mask multiplies the output of every expert."""
    from moe_routers_b200 import ops

    y = torch.ones(2 * 16, 64, dtype=torch.float16, device="cuda")
    y[16 + 3] = float("inf")
    idx = torch.zeros(16, 1, dtype=torch.int32, device="cuda")
    out = ops.combine_dense(y, idx, torch.ones(16, 1, device="cuda"), 2)
    assert torch.isnan(out[3]).all() and (out[torch.arange(16) != 3] == 1).all()


@pytest.mark.parametrize("bad", [-1, 4, 1 << 30])
def test_picks_of_experts_that_do_not_exist_are_reported(bad):
    """They add nothing, and the status of the stream says so."""
    from moe_routers_b200 import ops
    from moe_routers_b200._lib import MoeError

    y = torch.ones(4 * 40, 8, dtype=torch.bfloat16, device="cuda")
    idx = torch.tensor([[0, 3]], dtype=torch.int32, device="cuda").repeat(40, 1)
    gates = torch.tensor([[1.0, 2.0]], device="cuda").repeat(40, 1)
    assert (ops.combine_dense(y, idx, gates, 4) == 3).all() and ops.read_status() == 0
    idx[37, 1] = bad
    try:
        out = ops.combine_dense(y, idx, gates, 4)
        assert (out[37] == 1).all() and (out[torch.arange(40) != 37] == 3).all()
        with pytest.raises(MoeError, match="expert index"):
            ops.read_status()
    finally:  # the status block again as the other tests expect it
        ops.workspace(torch.device("cuda"), 1, 1, 1)[:4].zero_()
