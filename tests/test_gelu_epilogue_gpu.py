"""The grouped GEMM's GELU over the whole range of its argument: an identity weight hands every value to
the epilogue unchanged, so the stored result is the rounded GELU of an exactly known input."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gelu_epilogue_matches_double_precision(dtype):
    """Bound: half a unit in the last place of the storage type (2^-11 / 2^-8 of the value, fp16 subnormals
    2^-25 absolute; bf16 reaches below fp32's smallest normal number 2^-126, where the exponential is flushed to
    zero, and its factor 0.5 |v| t is at most 1.6 here: 2^-125) plus the epilogue's own 1e-5 relative error (its fp32 exponent argument reaches 36 before
    fp16 underflows, 36 * 2^-23 = 4.3e-6, with the fit's 3e-8 and two roundings of the special functions)."""
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
    eps, tiny = (2.0 ** -11, 2.0 ** -25) if dtype == torch.float16 else (2.0 ** -8, 2.0 ** -125)
    assert ((got - ref).abs() <= ref.abs() * (eps + 1e-5) + tiny).all()
