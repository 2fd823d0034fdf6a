"""The grouped GEMM's unit list: more units ahead than its ring holds, empty experts, the partial last round cut into
pieces of a unit's tokens, and column groups of 16 in the epilogue, against fp32 matrix products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(counts, k, n, dtype=torch.float16, act=None):
    from moe_routers_b200 import ops

    e, rows = len(counts), sum(counts)
    g = torch.Generator(device="cuda").manual_seed(rows * 31 + n)
    a = torch.empty(rows, k, dtype=dtype, device="cuda").normal_(generator=g)
    n_w = 2 * n if act == "swiglu" else n
    w = torch.empty(e, n_w, k, dtype=dtype, device="cuda").normal_(0.0, k ** -0.5, generator=g)
    ends = torch.tensor([0] + counts).cumsum(0)
    c = ops.grouped_gemm(a, w, ends.int().cuda(), activation=act)
    assert ops.read_status() == 0
    ref = torch.empty(rows, n, device="cuda")
    for i in range(e):
        r = a[ends[i]:ends[i + 1]].float() @ w[i].float().t()
        if act == "swiglu":
            r = torch.nn.functional.silu(r[:, :n]) * r[:, n:]
        elif act == "gelu":
            r = torch.nn.functional.gelu(r)
        ref[ends[i]:ends[i + 1]] = r
    # one rounding to 16 bits of values of up to about 6, and sums of k products in another order
    eps = 2.0 ** (-11 if dtype == torch.float16 else -8)
    torch.testing.assert_close(c.float(), ref, rtol=2 * eps, atol=1e-3 if dtype == torch.float16 else 4e-3)


@pytest.mark.parametrize("cnt", [1, 15, 16, 17, 31, 32, 33, 48, 49, 65])
@pytest.mark.parametrize("act", [None, "gelu", "swiglu"])
def test_column_groups(cnt, act):
    _check([cnt, 0, 2 * cnt, 1], 136, 144, act=act)


@pytest.mark.parametrize("experts,rows,n", [
    (1, 128, 256),       # one unit: two pieces
    (1, 127, 256),       # (with fewer than 128 rows there is one cluster per unit: whole)
    (1, 250, 5120),      # 20 units: three pieces each
    (1, 190, 6144),      # 24 units of 192 columns: three pieces each
    (1, 128, 4864),      # 19 units: three would fit, 128 columns give two
    (1, 250, 24064),     # 94 units: one full round and 20 in three pieces
    (1, 256, 4608),      # 18 units: four pieces each
    (1, 225, 4608),      # 18 units of 256 columns
    (1, 250, 9472),      # 37 units: two pieces
    (1, 250, 9728),      # 38 units: whole
    (1, 250, 18944),     # 74 units: one full round
    (1, 250, 19200),     # and one unit more, in four pieces
    (1, 600, 6400),      # 75 units of 224 and 192 columns
    (1, 96, 19200),      # a unit of fewer than 128 columns stays whole
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_partial_last_round(experts, rows, n, dtype):
    _check([rows] * experts, 192, n, dtype)


def test_many_units_and_empty_experts():
    _check([0, 300, 0, 0, 5, 257, 64, 0], 72, 9600, act="gelu")
    _check([0] * 40 + [3] + [0] * 900 + [70], 64, 64)
