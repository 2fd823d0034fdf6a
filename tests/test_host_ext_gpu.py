"""The host extension: its tensors are what torch.empty gives, its weight state is the tuple that it replaces,
and a changed, replaced or unregistered expert weight is still noticed by the layer."""
import struct

import pytest
import torch


def _layer(e=4):
    from moe_routers_b200.moe_layer import MoELayer

    return MoELayer(64, 64, e, 2)


def test_weight_state_follows_every_kind_of_change():
    from moe_routers_b200._host import weight_state
    from moe_routers_b200.moe_layer import SwiGLU

    names = ("w1", "w3", "w2")
    layer = _layer()
    state = lambda: weight_state(layer.experts._modules, names)  # noqa: E731
    params = [p for ex in layer.experts for p in (ex.w1.weight, ex.w3.weight, ex.w2.weight)]
    assert state() == b"".join(struct.pack("QQ", p.data_ptr(), p._version) for p in params)
    seen = [state()]
    with torch.no_grad():
        layer.experts[3].w3.weight.mul_(2)
    seen.append(state())
    layer.experts[1].w1.weight = torch.nn.Parameter(torch.randn(64, 64))
    seen.append(state())
    layer.experts[2] = SwiGLU(64, 64)
    seen.append(state())
    assert len(set(seen)) == 4
    del layer.experts[0].w2.weight
    layer.experts[0].w2.weight = torch.randn(64, 64)  # a plain tensor: looked up the long way
    assert state() is None


@pytest.mark.gpu
def test_empties_are_plain_tensors():
    from moe_routers_b200._host import empties

    a, b, c = empties(0, ((torch.int32, 3, 5), (torch.bfloat16, 7), (torch.float32, 0, 4)))
    assert a.shape == (3, 5) and a.dtype == torch.int32 and a.is_cuda and a.is_contiguous() and a.get_device() == 0
    assert b.shape == (7,) and b.dtype == torch.bfloat16 and c.numel() == 0
    assert len({t.untyped_storage().data_ptr() for t in (a, b)}) == 2
    with pytest.raises((RuntimeError, TypeError)):
        empties(0, ((torch.int32, -2),))


@pytest.mark.gpu
def test_empties_let_other_threads_run():
    """An allocation may wait for the device; a thread that has to launch the work it waits for must not be kept
    out meanwhile.  Many tensors in one call: nearly all of its time is the allocator's, and another thread's
    longest standstill stays well below it."""
    import threading
    import time

    from moe_routers_b200._host import empties

    specs = ((torch.uint8, 1),) * 200_000
    torch.empty(1, device="cuda")
    gaps, stop, running = [], threading.Event(), threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            now = time.perf_counter()
            gaps.append(now - last)
            last = now
            running.set()

    t = threading.Thread(target=tick)
    t.start()
    running.wait()
    begin = time.perf_counter()
    out = empties(0, specs)
    took = time.perf_counter() - begin
    stop.set()
    t.join()
    assert len(out) == len(specs)
    assert max(gaps) < 0.6 * took, (max(gaps), took)


@pytest.mark.gpu
def test_layer_sees_changed_weights():
    layer = _layer(8).half().cuda().requires_grad_(False)
    x = torch.randn(1, 16, 64, device="cuda").half()
    a = layer(x)
    for ex in layer.experts:
        ex.w2.weight.mul_(2)
    # doubling is exact but for results below fp16's normal range (spacing 2^-24), which are rounded before and
    # after the doubling: a row of them may move a sum of two by 2^-23, and that its rounding by one unit
    torch.testing.assert_close(layer(x), a * 2, rtol=2.0 ** -10, atol=2.0 ** -22)


@pytest.mark.gpu
def test_grouped_ffn_offsets_of_consecutive_calls():
    from moe_routers_b200 import grouped_ffn_cuda

    w = [torch.randn(64, 64, device="cuda").half() for _ in range(2)]
    for rows in ((3, 5), (8, 1), (1, 130)):
        a = [torch.randn(r, 64, device="cuda").half() for r in rows]
        for y, x, v in zip(grouped_ffn_cuda.grouped_ffn_forward(a, w), a, w):
            torch.testing.assert_close(y.float(), x.float() @ v.float(), rtol=2e-2, atol=2e-2)
