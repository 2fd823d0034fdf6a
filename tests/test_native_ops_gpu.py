"""The operators that the host extension runs as one call: the same results as the general Python path, which still takes
what is not plain and raises its errors."""
import pytest
import torch


def test_what_is_not_plain_is_left_alone():
    from moe_routers_b200 import _host, ops  # noqa: F401  (ops binds the entry points)

    x, w = torch.zeros(4, 64, dtype=torch.float16), torch.zeros(8, 64, dtype=torch.float16)
    assert _host.route(0, 0, x, w, 2, 0, 0.0, False) is None  # CPU tensors
    assert _host.route(0, 0, None, w, 2, 0, 0.0, False) is None
    assert _host.fused_select(0, 0, x, x, 64, 2) is None
    assert _host.sinkhorn(0, 0, True, x, 2, 10, 1e-6, 1.0) is None
    assert _host.grouped_lists(0, 0, [x], [w]) is None and _host.grouped_lists(0, 0, (), []) is None
    with pytest.raises(RuntimeError, match="inputs must be CUDA"):
        ops.route_fused(x, w, 2)


def _randn(*shape, dtype=torch.float16, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


def _strided(t):
    """The same values, not contiguous: the general path."""
    wide = torch.empty(*t.shape[:-1], 2 * t.size(-1), dtype=t.dtype, device=t.device)
    wide[..., ::2] = t
    return wide[..., ::2]


def _same(a, b):
    assert a.dtype == b.dtype and a.shape == b.shape and a.is_contiguous() and torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("t,d,e,k,dtype", [(1, 64, 8, 1, torch.float16), (33, 520, 60, 4, torch.bfloat16), (300, 128, 256, 8, torch.float16)])
def test_routes(t, d, e, k, dtype):
    from moe_routers_b200 import ops

    x, w = _randn(t, d, dtype=dtype), _randn(e, d, dtype=dtype, seed=1)
    for kw in (dict(), dict(skew_experts=min(4, e), skew_bias=2.0, return_logits=True)):
        a, b = ops.route_fused(x, w, k, **kw), ops.route_fused(_strided(x), _strided(w), k, **kw)
        assert list(a) == list(b) and a["workspace"] is b["workspace"]
        for name in a:
            if name != "workspace":
                _same(a[name], b[name])
    logits = _randn(t, e, seed=2)
    for a, b in zip(ops.fused_select(logits, x, e, k), ops.fused_select(_strided(logits), x, e, k)):
        _same(a, b)
    for fn in (ops.sinkhorn, ops.sinkhorn_router):
        for a, b in zip(fn(logits, k, iters=3), fn(_strided(logits), k, iters=3)):
            _same(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("act,t,k", [("gelu", 40, 2), ("swiglu", 5, 4), (None, 300, 1)])
def test_expert_ffn(act, t, k):
    from moe_routers_b200 import ops

    e, d, h = 8, 128, 192
    o = ops.route_fused(_randn(t, d), _randn(e, d, seed=1), k)
    w1, w2 = _randn(e, 2 * h if act == "swiglu" else h, d, seed=2) / 8, _randn(e, d, h, seed=3) / 8
    a = ops.expert_ffn(o["packed"], w1, w2, o["offsets"], o["gates"], o["route_row"], k, activation=act)
    hid = ops.grouped_gemm(o["packed"], w1, o["offsets"], activation=act)
    _same(a, ops.combine(ops.grouped_gemm(hid, w2, o["offsets"]), o["gates"], o["route_row"], k))
    _same(a, ops.expert_ffn(o["packed"], _strided(w1), w2, o["offsets"].long(), o["gates"], o["route_row"], k, activation=act))


@pytest.mark.gpu
def test_expert_ffn_with_an_odd_number_of_swiglu_features():
    """Gate and up rows are the first 2 h of an expert's 2 h + 1; the last one is not used."""
    from moe_routers_b200 import ops

    e, d, h, k = 4, 128, 64, 2
    o = ops.route_fused(_randn(24, d), _randn(e, d, seed=1), k)
    w1, w2 = _randn(e, 2 * h + 1, d, seed=2) / 8, _randn(e, d, h, seed=3) / 8
    args = o["offsets"], o["gates"], o["route_row"], k
    _same(ops.expert_ffn(o["packed"], w1, w2, *args, activation="swiglu"),
          ops.expert_ffn(o["packed"], w1[:, :2 * h].contiguous(), w2, *args, activation="swiglu"))


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[5], [0, 3, 0, 70, 1], [1] * 100, [2, 0] * 300])
def test_grouped_lists(counts):
    from moe_routers_b200 import grouped_ffn_cuda, ops

    e, kd, n = len(counts), 72, 64
    pool = _randn(sum(counts) + 9, kd)
    kn = _randn(e + 1, kd, n, seed=1) / 8
    ins, ws = list(torch.split(pool[4:4 + sum(counts)], counts)), list(kn[1:].unbind(0))
    out = ops.grouped_lists(ins, ws)
    assert isinstance(out, list) and [o.shape for o in out] == [(c, n) for c in counts]
    apart = [i.clone() for i in ins]
    assert e == 1 or ops.grouped_lists(apart, ws) is None  # not one buffer: the general path
    for a, b in zip(out, grouped_ffn_cuda.grouped_ffn_forward(apart, ws)):
        _same(a, b)
    _same(torch.cat(out), torch.cat(grouped_ffn_cuda.grouped_ffn_forward(ins, ws)))
    assert ops.grouped_lists(ins, [w.t() for w in ws]) is None and ops.grouped_lists(ins, ws[:-1]) is None
    assert ops.read_status() == 0


@pytest.mark.gpu
def test_grouped_lists_holds_its_buffers(monkeypatch):
    """Whoever empties the lists during the call (here the code that makes the scratch buffer, in a program another thread)
    does not take the rows and weights away from it."""
    from moe_routers_b200 import ops

    a, w = _randn(12, 64), _randn(4, 64, 64, seed=1) / 8
    want = torch.cat(ops.grouped_lists(list(a.clone().split(3)), list(w.clone().unbind(0))))
    ins, ws, spoiled, stream = list(a.clone().split(3)), list(w.clone().unbind(0)), [], ops._stream

    def meanwhile():
        ins.clear(), ws.clear()
        spoiled.extend(torch.full_like(t, float("nan")) for t in (a, w) for _ in range(4))  # what was given back is taken
        return stream()

    ops._workspaces.pop((torch.cuda.current_device(), stream()), None)
    monkeypatch.setattr(ops, "_stream", meanwhile)
    out = ops.grouped_lists(ins, ws)
    monkeypatch.undo()
    assert spoiled
    _same(torch.cat(out), want)


@pytest.mark.gpu
def test_errors_are_those_of_the_general_path():
    from moe_routers_b200 import ops
    from moe_routers_b200._lib import MoeError

    x, w = _randn(4, 64), _randn(8, 64, seed=1)
    with pytest.raises(MoeError, match="top_k"):
        ops.route_fused(x, w, 9)
    with pytest.raises(RuntimeError, match="fp16"):
        ops.route_fused(x, w.float(), 2)
    with pytest.raises(RuntimeError, match="router weight must be"):
        ops.route_fused(x, _randn(8, 56), 2)
    with pytest.raises(MoeError, match="epsilon"):
        ops.sinkhorn(x, 2, epsilon=0.0)
    with pytest.raises(MoeError, match="n_experts"):
        ops.fused_select(_randn(4, 4), x, 4, 8)
    for logits in (_randn(3, 8), _randn(4, 7)):
        with pytest.raises(RuntimeError, match="logits must be"):
            ops.fused_select(logits, x, 8, 2)
    for a, b in zip(ops.fused_select(w.view(4, 128)[:, :8].reshape(2, 16), x, 8, 2), ops.fused_select(w[::2, :8], x, 8, 2)):
        _same(a, b)  # as many in another shape: row by row
    for a, b in zip(ops.fused_select(torch.cat([w[:, :8], w[:, 8:16]])[:9], x, 8, 2), ops.fused_select(w[:4, :8], x, 8, 2)):
        _same(a, b)  # more logits than tokens: the first ones, as ever
    o = ops.route_fused(x, w, 2)
    for name, short, text in (("offsets", o["offsets"][:8], "offsets must have"), ("gates", o["gates"][:3], "gates must be"),
                              ("gates", o["gates"].repeat(1, 2), "gates must be"), ("route_row", o["route_row"][:7], "route_row must")):
        r = {**o, name: short}
        with pytest.raises(RuntimeError, match=text):
            ops.expert_ffn(r["packed"], _randn(8, 64, 64), _randn(8, 64, 64), r["offsets"], r["gates"], r["route_row"], 2, activation=None)
    with pytest.raises(RuntimeError, match="inner dimensions"):
        ops.expert_ffn(o["packed"], _randn(8, 64, 32), w.view(8, 8, 8), o["offsets"], o["gates"], o["route_row"], 2, activation=None)
