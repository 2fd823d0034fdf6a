"""The grouped GEMM's GELU over the whole range of its argument: an identity weight hands every value to
the epilogue unchanged, so the stored result is the rounded GELU of an exactly known input."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gelu_epilogue_matches_double_precision(dtype):
    """0.5 v (1 + erff(v / sqrt 2)) in fp32.  Bound: half a unit in the last place of the storage type (2^-11 /
    2^-8 of the value, fp16 subnormals 2^-25 absolute), two products (2^-23 of the value), and 0.5 |v| times the
    error of the bracket: erff's 2 ulp (2^-23), its rounded argument (z erf'(z) <= 0.5 times 2^-23) and the rounded
    sum (2^-24), 2^-22 together."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from moe_routers_b200 import ops

    K = 64
    v = torch.cat([torch.linspace(-14, 14, 16000), torch.tensor([0.0, -0.0, 1e-4, -1e-4, 60000.0, -60000.0])])
    v = torch.nn.functional.pad(v, (0, -v.numel() % K)).to(dtype).view(-1, K).cuda()
    eye = torch.eye(K, dtype=dtype, device="cuda").unsqueeze(0)
    off = torch.tensor([0, v.size(0)], dtype=torch.int32, device="cuda")
    got = ops.grouped_gemm(v, eye, off, layout="nk", activation="gelu").double()
    x = v.double()
    ref = 0.5 * x * torch.special.erfc(-x / 2 ** 0.5)
    eps, tiny = (2.0 ** -11, 2.0 ** -25) if dtype == torch.float16 else (2.0 ** -8, 0.0)
    assert ((got - ref).abs() <= ref.abs() * (eps + 2.0 ** -22) + x.abs() * 2.0 ** -23 + tiny).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gelu_epilogue_special_values(dtype):
    """What 0.5 v (1 + erf) gives: -inf * 0 is NaN, and nothing is left of a value whose 1 + erf is 0 in fp32.  The
    bias hands each value to the epilogue; the product in front of it is 0."""
    from moe_routers_b200 import ops

    inf, nan = float("inf"), float("nan")
    v = torch.tensor([inf, -inf, nan, -nan, -8.0, -1e4, 1e4, 0.0]).to(dtype)
    K = 64
    bias = torch.nn.functional.pad(v, (0, K - v.numel())).view(1, K).cuda()
    a = torch.zeros(3, K, dtype=dtype, device="cuda")
    w = torch.zeros(1, K, K, dtype=dtype, device="cuda")
    off = torch.tensor([0, 3], dtype=torch.int32, device="cuda")
    got = ops.grouped_gemm(a, w, off, layout="nk", activation="gelu", bias=bias)
    assert ops.read_status() == 0
    want = torch.tensor([inf, nan, nan, nan, 0.0, 0.0, 1e4, 0.0]).to(dtype)
    torch.testing.assert_close(got[:, :8].cpu(), want.expand(3, 8), rtol=0, atol=0, equal_nan=True)
