"""The route of a small batch in one launch (at most 32 tokens and two 2 KB pieces per warp of the cluster), at
its edges and just past them, against the two-launch form (the pack of the same selection)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [1, 2, 8, 9, 10, 11, 16, 20, 21, 31, 32, 33])
@pytest.mark.parametrize("d,e,k,dtype", [(8, 3, 1, torch.float16), (72, 16, 2, torch.bfloat16), (520, 60, 8, torch.float16),
                                         (1032, 64, 2, torch.bfloat16), (4096, 64, 2, torch.float16),
                                         (8192, 256, 8, torch.bfloat16)])
def test_one_launch_route(t, d, e, k, dtype):
    from moe_routers_b200 import ops
    from moe_routers_b200._lib import lib

    g = torch.Generator().manual_seed(t * 31 + d)
    x = torch.randn(t, d, generator=g).to(dtype).cuda()
    w = (torch.randn(e, d, generator=g) / d ** 0.5).to(dtype).cuda()
    before = lib.moe_launch_count()
    o = ops.route_fused(x, w, k, skew_experts=2, skew_bias=0.5)
    slices = 4 if d > 960 else 2 if d > 192 else 1
    one = t <= 32 and t * k <= 64 and t * -(-d // 1024) <= 2 * 10 * slices
    assert lib.moe_launch_count() - before == (1 if one else 2)
    for _ in range(3):  # back to back, into fresh buffers
        o = ops.route_fused(x, w, k, skew_experts=2, skew_bias=0.5)
    idx, gates = ops.router_gemm_select(x, w, k, skew_experts=2, skew_bias=0.5)
    counts, offsets, packed, row_route, route_row = ops.pack(x, idx, e)
    want = dict(idx=idx, gates=gates, counts=counts, offsets=offsets, packed=packed, row_route=row_route, route_row=route_row)
    for name, ref in want.items():
        assert torch.equal(o[name], ref), name
    assert torch.equal(o["packed"], x[(o["row_route"] // k).long()])
    # the histograms are left for the scatter half
    fresh = dict(o, packed=torch.zeros_like(packed))
    o2 = ops.route_fused(x, w, k, skew_experts=2, skew_bias=0.5)
    ops.pack_scatter(x, e, dict(fresh, workspace=o2["workspace"]))
    assert torch.equal(fresh["packed"], packed)
    assert ops.read_status() == 0


def test_one_launch_route_unaligned_packed():
    from moe_routers_b200 import ops

    x = torch.randn(7, 64, device="cuda").half()
    w = torch.randn(8, 64, device="cuda").half()
    o = ops.route_fused(x, w, 2)
    out = dict(o, packed=torch.zeros(14 * 64 + 1, dtype=torch.float16, device="cuda")[1:].view(14, 64))
    ops.route_fused(x, w, 2, out=out)  # 2 bytes off: the scatter kernel's word copies
    assert torch.equal(out["packed"], o["packed"])
