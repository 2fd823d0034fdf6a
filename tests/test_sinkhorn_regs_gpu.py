"""The Sinkhorn kernel that keeps the matrix in registers, at the edges of its layouts: columns per lane,
rows per lane, CTAs per cluster, and the shapes just outside of it, against the reference's iteration
(models/decoder_moe.py:92-123) in 64 bits."""
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
    (100, 257, 2, 10, torch.float32),
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
    # the router's own result types are these values, rounded once
    ridx, rw = SinkhornRouter(iters=iters)(logits, k)
    assert ridx.dtype == torch.int64 and rw.dtype == dtype
    assert torch.equal(ridx, idx.long()) and torch.equal(rw, w.to(dtype))


def test_sinkhorn_unaligned_logits():
    from moe_routers_b200 import ops

    g = torch.Generator().manual_seed(5)
    flat = torch.randn(300 * 64 + 1, generator=g).half().cuda()
    a = flat[1:].view(300, 64)  # rows 2 bytes off a 16-byte boundary
    b = a.clone()
    for x, y in zip(ops.sinkhorn(a, 4), ops.sinkhorn(b, 4)):
        assert torch.equal(x, y)
