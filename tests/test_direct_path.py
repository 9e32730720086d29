"""The direct launch path of plain eager calls: taken only there, and equal to the custom ops."""

import threading
import time

import pytest
import torch
import torch.utils.checkpoint

from kohakufa_b200 import _lib, attention, attention_varlen, pack_mask, set_backward, varlen_plan
from kohakufa_b200 import op


def test_plain_eager_is_plain():
    t = torch.ones(2)
    assert _lib.plain_eager(t, t)
    assert not _lib.plain_eager(t, torch.nn.Parameter(t))

    class Sub(torch.Tensor):
        pass

    assert not _lib.plain_eager(t.as_subclass(Sub))
    seen = []

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class FunctionMode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert not _lib.plain_eager(t)
    with FunctionMode():
        assert not _lib.plain_eager(t)
    with torch.autograd.forward_ad.dual_level():
        assert not _lib.plain_eager(t)
    torch.func.vmap(lambda x: (seen.append(_lib.plain_eager(x)), x)[1])(t)
    torch.func.grad(lambda x: (seen.append(_lib.plain_eager(x)), x.sum())[1])(t)
    torch.jit.trace(lambda x: (seen.append(_lib.plain_eager(x)), x + 1)[1], t, check_trace=False)
    assert seen == [False, False, False]
    assert _lib.plain_eager(t)


def test_plain_eager_leaves_to_the_dispatcher_what_it_resolves():
    t = torch.ones(3, 2)
    assert not _lib.plain_eager(torch._neg_view(t)) and not _lib.plain_eager(t, torch._efficientzerotensor(2))
    seen = []

    class Double(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return 2 * x

        @staticmethod
        def backward(ctx, g):
            seen.append(_lib.plain_eager(g))
            return 2 * g

    x = torch.ones(2, requires_grad=True)
    torch.autograd.grad(Double.apply(x), x, t, is_grads_batched=True)
    assert seen == [False]
    assert _lib.plain_eager(t, x)


def test_sequence_offsets_are_refused_before_a_launch():
    """The kernels read the offsets where they lie: int32, contiguous, on the device of q, as many for q as for k."""
    host, t = _lib.host(), torch.zeros(4, 1, 16, dtype=torch.float16)
    lse, word = torch.zeros(1, 1, 2, 4), torch.zeros(1, dtype=torch.int32)
    cu = torch.tensor([0, 4], dtype=torch.int32)
    strided = torch.tensor([[0, 9], [4, 9]], dtype=torch.int32)[:, 0]
    for bad in (strided, cu.long(), cu.to("meta"), cu[:1], torch.tensor([0, 2, 4], dtype=torch.int32)):
        for pair in ((bad, cu), (cu, bad)):
            with pytest.raises(ValueError, match="cu_seqlens"):
                host.forward_varlen(t, t, t, *pair, 4, 4, 1.0, 0, word)
            with pytest.raises(ValueError, match="cu_seqlens"):
                host.backward_varlen(t, t, t, t, t, lse, *pair, 4, 4, 1.0, 0, word)
    with pytest.raises(ValueError, match="different devices"):
        host.forward_varlen(t, t.to("meta"), t, cu, cu, 4, 4, 1.0, 0, word)


def inputs(dim=128, seq=200, heads=4, kv_heads=2, packed=False):
    gen = torch.Generator().manual_seed(dim + seq)
    shape = (seq, heads, dim) if packed else (2, seq, heads, dim)
    kv_shape = (seq, kv_heads, dim) if packed else (2, seq, kv_heads, dim)
    ts = [torch.randn(s, generator=gen).bfloat16().cuda() for s in (shape, kv_shape, kv_shape, shape)]
    if not packed:
        ts = [t.transpose(1, 2) for t in ts]
    return [t.requires_grad_() for t in ts[:3]], ts[3]


def both_ways(call, qkv, dout, monkeypatch):
    """(out, dq, dk, dv) of the direct path and of the custom ops."""
    results = []
    for direct in (True, False):
        with monkeypatch.context() as m:
            if not direct:
                m.setattr(_lib, "plain_eager", lambda *ts: False)
            out = call(*qkv)
            assert ("sm100" in type(out.grad_fn).__name__) == (not direct)
            results.append([out.detach(), *torch.autograd.grad(out, qkv, dout)])
            with torch.no_grad():
                assert torch.equal(call(*qkv), out)
    return results


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "mask", "varlen"])
def test_direct_path_equals_the_ops(kind, monkeypatch):
    (q, k, v), dout = inputs(packed=kind == "varlen")
    if kind == "mask":
        mask = (torch.rand(200, 200, generator=torch.Generator().manual_seed(1)) < 0.4).cuda()
        call = lambda q, k, v: attention(q, k, v, mask=mask)  # noqa: E731
    elif kind == "varlen":
        cu = torch.tensor([0, 70, 200], dtype=torch.int32, device="cuda")
        plan = varlen_plan(cu, cu)
        call = lambda q, k, v: attention_varlen(q, k, v, cu, cu, causal=True, plan=plan)  # noqa: E731
    else:
        call = lambda q, k, v: attention(q, k, v, causal=True)  # noqa: E731
    direct, ops = both_ways(call, (q, k, v), dout, monkeypatch)
    for a, b in zip(direct, ops):
        assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride()
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_direct_path_and_autograd_features():
    (q, k, v), dout = inputs()
    out = attention(q, k, v)
    want = torch.autograd.grad(out, (q, k, v), dout)
    with torch.autograd.graph.save_on_cpu():  # saved tensors leave the GPU and come back with other strides
        out = attention(q, k, v)
    for a, b in zip(torch.autograd.grad(out, (q, k, v), dout), want):
        assert torch.equal(a, b)
    out = attention(q, k, v)  # an expanded gradient has strides of 0
    grads = torch.autograd.grad(out.sum(), (q, k, v))
    ones = torch.autograd.grad(attention(q, k, v), (q, k, v), torch.ones_like(out))
    assert all(torch.equal(a, b) for a, b in zip(grads, ones))
    (dq,) = torch.autograd.grad(attention(q, k, v), (q,), dout, create_graph=True)
    with pytest.raises(RuntimeError):  # there is no second derivative
        torch.autograd.grad(dq.sum(), (q,))
    out = attention(q, k, v)
    with torch.no_grad():
        q.mul_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(dout)


@pytest.mark.gpu
def test_recorded_calls_in_the_engine():
    """The node's backward runs on a thread of the autograd engine: an error of the library there is the exception a direct
    call raises, a checkpoint's recomputation (which leaves the forward by an exception of a saved-tensor hook) works, and
    so does a backward that finds a dispatch mode (the registered op runs)."""
    (q, k, v), dout = inputs()
    out = attention(q, k, v)
    flat = torch.empty(dout.numel() + 8, dtype=dout.dtype, device="cuda")[1 : dout.numel() + 1]
    odd = flat.copy_(dout.transpose(1, 2).reshape(-1)).view(2, 200, 4, 128).transpose(1, 2)  # starts 2 bytes past a boundary
    with pytest.raises(_lib.KfaError):
        torch.autograd.grad(out, (q, k, v), odd, retain_graph=True)
    want = torch.autograd.grad(out, (q, k, v), dout)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out, (q, k, v), dout)
    out = torch.utils.checkpoint.checkpoint(attention, q, k, v, use_reentrant=False)
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(out, (q, k, v), dout), want))
    seen = []

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func.name())
            return func(*args, **(kwargs or {}))

    out = attention(q, k, v)
    with Mode():
        got = torch.autograd.grad(out, (q, k, v), dout)
    assert "kohakufa_b200::sm100_backward" in seen
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dim", [("plain", 128), ("plain", 48), ("plain", 40), ("mask", 128), ("varlen", 128)])
def test_batched_gradients(kind, dim):
    """``is_grads_batched`` gives the rows of one call per gradient (the split kernels repeat bit for bit)."""
    (q, k, v), dout = inputs(dim, packed=kind == "varlen")
    if kind == "varlen":
        cu = torch.tensor([0, 70, 200], dtype=torch.int32, device="cuda")
        out = attention_varlen(q, k, v, cu, cu)
    else:
        out = attention(q, k, v, mask=torch.ones(200, 200, dtype=torch.bool, device="cuda") if kind == "mask" else None)
    douts = torch.stack([dout, -dout, 2 * dout])
    got = torch.autograd.grad(out, (q, k, v), douts, is_grads_batched=True, retain_graph=True)
    for i, g in enumerate(douts):
        for a, b in zip(got, torch.autograd.grad(out, (q, k, v), g, retain_graph=True)):
            assert torch.equal(a[i], b)


@pytest.mark.gpu
def test_negative_views():
    (q, k, v), dout = inputs()
    with torch.no_grad():
        assert torch.equal(attention(torch._neg_view(q), k, v), attention(-q, k, v))
    out = attention(q, k, v)
    got = torch.autograd.grad(out, (q, k, v), torch._neg_view(dout), retain_graph=True)
    assert all(torch.equal(a, b) for a, b in zip(got, torch.autograd.grad(out, (q, k, v), -dout)))


@pytest.mark.gpu
def test_sequence_offsets_of_a_table():
    """A column of a 2-D table is taken (as if it were contiguous); offsets in host memory are refused."""
    (q, k, v), _ = inputs(packed=True)
    table = torch.tensor([[0, 5], [70, 6], [200, 7]], dtype=torch.int32, device="cuda")
    cu = table[:, 0].contiguous()
    with torch.no_grad():
        assert torch.equal(attention_varlen(q, k, v, table[:, 0], table[:, 0]), attention_varlen(q, k, v, cu, cu))
        with pytest.raises(ValueError, match="cu_seqlens"):
            attention_varlen(q, k, v, cu.cpu(), cu.cpu())


@pytest.mark.gpu
def test_other_threads_run_while_launches_wait():
    """With the stream busy and its queue full a launch waits for the device; Python's other threads do not."""
    q, k, v = (torch.randn(1, 1, 64, 64, device="cuda").half() for _ in range(3))
    attention(q, k, v)
    ticks, done = [], threading.Event()

    def tick():
        while not done.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    thread = threading.Thread(target=tick)
    thread.start()
    torch.cuda._sleep(int(1.2e9))  # more than half a second at any clock of the GPU
    start = time.perf_counter()
    for _ in range(2500):  # the queue holds about 1000 launches
        attention(q, k, v)
    waited = time.perf_counter() - start
    torch.cuda.synchronize()
    done.set()
    thread.join()
    assert waited > 0.4
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < 0.2


@pytest.mark.gpu
def test_direct_path_refuses_what_the_ops_refuse():
    (q, k, v), _ = inputs()
    for bad, error in (((q.float(), k, v), TypeError), ((q, k[:, :1], v), ValueError), ((q[:, :3], k, v), ValueError),
                       ((q.mT, k.mT, v.mT), ValueError), ((q.cpu(), k.cpu(), v.cpu()), ValueError)):  # fmt: skip
        with pytest.raises(error):
            op.attention(*bad)
    packed = pack_mask(torch.ones(100, 200, dtype=torch.bool, device="cuda"), 2, 4, 100, 200)
    with pytest.raises(ValueError):
        op.attention(q, k, v, mask=packed)
    set_backward("auto")
