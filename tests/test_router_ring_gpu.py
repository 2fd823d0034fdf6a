"""The router kernel's partial tiles in the pipeline ring (E >= 128), at the expert counts where the layout
changes, against the selection from the logits that the kernel itself reports and an fp32 product."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [112, 113, 128, 129, 144, 145, 192, 193, 208, 240, 241, 256])
@pytest.mark.parametrize("t,d,k", [(1, 64, 1), (129, 200, 2), (300, 1024, 8), (2049, 2048, 4)])
def test_ring_layouts(t, d, k, e):
    from moe_routers_b200 import ops

    g = torch.Generator().manual_seed(t + d + e)
    x = torch.randn(t, d, generator=g).half().cuda()
    w = (torch.randn(e, d, generator=g) / d ** 0.5).half().cuda()
    for _ in range(3):  # back to back: a launch may start under the one before
        o = ops.route_fused(x, w, k, return_logits=True)
    assert ops.read_status() == 0
    # fp32 sums of products of 16-bit values, rounded once to fp16: half a unit plus the sums' own rounding
    torch.testing.assert_close(o["logits"], x.float() @ w.float().t(), rtol=2.0 ** -10, atol=2.0 ** -12)
    idx, gates, _ = oracle.topk_select(o["logits"].cpu().numpy(), k)
    np.testing.assert_array_equal(o["idx"].cpu().numpy(), idx.astype(np.int32))
    np.testing.assert_allclose(o["gates"].cpu().numpy(), gates, rtol=1e-5, atol=1e-7)
    assert torch.equal(o["packed"], x[(o["row_route"] // k).long()])
