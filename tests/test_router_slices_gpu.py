"""The router kernel at the batch sizes where a CTA takes one, two or four slices of K: the logits of a token do
not depend, to the last bit, on how many tokens come with it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,e,k,dtype", [(64, 8, 2, torch.float16), (256, 16, 2, torch.bfloat16), (1000, 64, 2, torch.float16),
                                         (1032, 60, 4, torch.bfloat16), (2048, 64, 8, torch.float16),
                                         (1088, 96, 2, torch.float16), (1024, 128, 4, torch.bfloat16), (512, 256, 2, torch.float16)])
def test_logits_do_not_depend_on_the_batch(d, e, k, dtype):
    from moe_routers_b200 import ops

    g = torch.Generator().manual_seed(d + e)
    x = torch.randn(19100, d, generator=g).to(dtype).cuda()
    w = (torch.randn(e, d, generator=g) / d ** 0.5).to(dtype).cuda()
    ref = torch.cat([ops.router_gemm_select(c.contiguous(), w, k, return_logits=True)[2] for c in x.split(1024)])
    eps = 2.0 ** (-11 if dtype == torch.float16 else -8)
    torch.testing.assert_close(ref, x.float() @ w.float().t(), rtol=2 * eps, atol=2.0 ** -12)
    for t in (4736, 4737, 9472, 9473, 18944, 18945, 19100):
        idx, gates, logits = ops.router_gemm_select(x[:t], w, k, return_logits=True)
        assert torch.equal(logits, ref[:t]), t
        top = torch.topk(logits, k).values
        assert torch.equal(torch.gather(logits, 1, idx.long()), top), t
    assert ops.read_status() == 0
