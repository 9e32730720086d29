"""Head dims that are odd multiples of 8, computed without widening the tensors: against the zero-padded path,
whose kernels do the same arithmetic on the same values."""

import pytest
import torch

from kohakufa_b200 import _lib, attention, op, set_backward

pytestmark = pytest.mark.gpu


def inputs(dim, s_q, s_kv, heads, kv_heads, dtype, layout):
    gen = torch.Generator().manual_seed(dim + s_q)

    def one(seq, h):
        if layout == "bshd":
            return torch.randn(2, seq, h, dim, generator=gen).to(dtype).cuda().transpose(1, 2)
        if layout == "bhsd":
            return torch.randn(2, h, seq, dim, generator=gen).to(dtype).cuda()
        wide = torch.randn(2, seq, h, dim + 8, generator=gen).to(dtype).cuda()  # columns 8 .. of wider rows
        return wide[..., 8:].transpose(1, 2)

    q, k, v, dout = one(s_q, heads), one(s_kv, kv_heads), one(s_kv, kv_heads), one(s_q, heads)
    return [t.detach().requires_grad_() for t in (q, k, v)], dout


@pytest.mark.parametrize("dim", [8, 24, 40, 56, 72, 88, 104, 120])
@pytest.mark.parametrize("layout", ["bshd", "bhsd", "sliced"])
@pytest.mark.parametrize("s_q,s_kv,mode", [(1, 1, {}), (129, 77, {}), (300, 300, {"causal": True}), (257, 400, {"block_causal": 100})])
def test_narrow_equals_padded(dim, layout, s_q, s_kv, mode, monkeypatch):
    """Equal bits: zero columns add exact zeros to every product. (The split backward, whose dQ repeats.)"""
    dtype = torch.float16 if dim % 3 else torch.bfloat16
    qkv, dout = inputs(dim, s_q, s_kv, 4, 2, dtype, layout)
    results = []
    set_backward("split")
    try:
        for narrow in (True, False):
            with monkeypatch.context() as m:
                if narrow:
                    assert op.narrow(*qkv)
                else:
                    m.setattr(op, "narrow", lambda *ts: False)
                out = attention(*qkv, **mode)
                results.append([out, *torch.autograd.grad(out, qkv, dout)])
    finally:
        set_backward("auto")
    assert _lib.device_status() == 0
    for a, b in zip(*results):
        assert a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.parametrize("dim", [56, 120])
def test_narrow_fused_backward(dim):
    """dQ is summed by fp32 adds in no fixed order: against the split kernels at the tolerance of those adds."""
    qkv, dout = inputs(dim, 300, 300, 4, 2, torch.bfloat16, "bshd")
    grads = {}
    try:
        for mode in ("split", "fused"):
            set_backward(mode)
            grads[mode] = torch.autograd.grad(attention(*qkv, causal=True), qkv, dout)
    finally:
        set_backward("auto")
    for a, b in zip(grads["fused"], grads["split"]):
        assert float((a.double() - b.double()).norm() / b.double().norm()) < 5e-3


def test_narrow_leaves_other_inputs_alone():
    (q, k, v), _ = inputs(40, 64, 64, 4, 4, torch.float16, "bshd")
    assert not op.narrow(q[..., :36], k[..., :36], v[..., :36])  # no multiple of 8
    flat = torch.randn(2, 64, 4 * 40 + 4).half().cuda()[..., :160].unflatten(-1, (4, 40)).transpose(1, 2)
    assert not op.narrow(flat, k, v)  # rows that do not start on 16 bytes
    assert attention(flat, k, v).shape == flat.shape
    shifted = torch.randn(2 * 64 * 4 * 40 + 4).half().cuda()[4:].view(2, 64, 4, 40).transpose(1, 2)  # starts on 8 bytes
    assert not op.narrow(q, shifted, v) and not op.narrow(shifted, k, v)
    assert attention(q, shifted, v).shape == q.shape
    want = torch.autograd.grad(attention(q, k, v), (q, k, v), shifted.contiguous())
    for a, b in zip(torch.autograd.grad(attention(q, k, v), (q, k, v), shifted), want):
        assert float((a - b).float().norm()) <= 1e-3 * float(b.float().norm())
    for bad in (lambda: op.attention(q, k, v), lambda: attention(q, k[:, :3], v[:, :3])):
        with pytest.raises(ValueError):
            bad()


def test_long_recorded_calls_are_widened():
    """Where the backward's reads of narrow rows cost more than the copies: only calls that autograd records."""
    q = torch.zeros(1, 20000, 1, 104, dtype=torch.float16, device="cuda").transpose(1, 2)
    assert op.narrow(q, q, q)
    leaf = q.detach().requires_grad_()
    assert not op.narrow(leaf, q, q) and op.narrow(leaf[:, :, :1000], q[:, :, :1000], q[:, :, :1000])
    with torch.no_grad():
        assert op.narrow(leaf, q, q)
