"""The bulk scatter at token counts around its splits (tiles shared by up to 8 CTAs, whole tiles, halved tiles with three CTAs
per SM), at many routes per tile and with short and long rows, against the canonical pack."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,d,e,k", [
    (1, 8, 4, 1), (7, 4096, 8, 2), (33, 64, 64, 8), (64, 5000, 16, 2), (147, 1032, 60, 4), (148, 512, 8, 1), (149, 512, 8, 2),
    (295, 2048, 256, 8), (1000, 72, 128, 6), (4736, 264, 64, 2), (4737, 256, 60, 2), (4750, 1024, 60, 2), (7104, 4112, 16, 2), (7105, 136, 64, 8), (9473, 128, 32, 8),
    (16387, 96, 64, 2), (16387, 8, 256, 4), (33000, 16, 300, 1)])
def test_rows_and_maps(t, d, e, k):
    from moe_routers_b200 import ops

    g = torch.Generator().manual_seed(t + d)
    x = torch.randint(-30000, 30000, (t, d), generator=g, dtype=torch.int16)
    idx = torch.stack([torch.randperm(e, generator=g)[:k] for _ in range(min(t, 512))]).repeat(-(-t // 512), 1)[:t].int()
    idx[t // 2:] = idx[t // 2:].clamp_max(max(k - 1, e // 3))  # repeated picks, uneven experts
    packed, counts, offsets, row_route, route_row = oracle.pack_canonical(x.numpy(), idx.numpy(), e)
    got = ops.pack(x.view(torch.float16).cuda(), idx.cuda(), e)
    assert ops.read_status() == 0
    for a, b in zip(got, (counts, offsets, packed, row_route, route_row)):
        a = a.view(torch.int16) if a.dtype == torch.float16 else a
        np.testing.assert_array_equal(a.cpu().numpy(), b)
    plan = ops.pack(x.view(torch.float16).cuda(), idx.cuda(), e, copy_rows=False)  # the maps without the rows
    for a, b in zip((plan[0], plan[1], plan[3], plan[4]), (counts, offsets, row_route, route_row)):
        np.testing.assert_array_equal(a.cpu().numpy(), b)
