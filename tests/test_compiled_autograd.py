"""A graph that eager calls recorded, under compiled autograd: the backward is compiled without a break, through the registered
ops."""

import pytest
import torch
from torch._dynamo import compiled_autograd

from kohakufa_b200 import attention, attention_varlen, set_backward, varlen_plan

pytestmark = pytest.mark.gpu


def recorded(kind, dim, seq):
    gen = torch.Generator().manual_seed(dim + seq)
    shape = (seq, 4, dim) if kind == "varlen" else (2, 4, seq, dim)
    leaves = [torch.randn(shape, generator=gen).half().cuda().requires_grad_() for _ in range(3)]
    if kind == "varlen":
        cu = torch.tensor([0, 70, seq], dtype=torch.int32, device="cuda")
        out = attention_varlen(*leaves, cu, cu, causal=True, plan=varlen_plan(cu, cu))
    else:
        mask = (torch.rand(seq, seq, generator=gen) < 0.4).cuda() if kind == "mask" else None
        out = attention(*leaves, mask=mask)
    return out, leaves, torch.randn(out.shape, generator=gen).half().cuda()


@pytest.mark.parametrize("dynamic", [False, True])
@pytest.mark.parametrize("kind,dim", [("plain", 128), ("plain", 64), ("plain", 40), ("mask", 128), ("varlen", 128)])
def test_a_recorded_graph_is_compiled_whole(kind, dim, dynamic):
    torch._dynamo.reset()
    set_backward("split")  # (repeats bit for bit)
    try:
        for seq in (200, 328):
            out, leaves, dout = recorded(kind, dim, seq)
            want = torch.autograd.grad(out, leaves, dout, retain_graph=True)
            with compiled_autograd._enable(lambda gm: torch.compile(gm, backend="aot_eager", fullgraph=True, dynamic=dynamic)):
                out.backward(dout)
            assert all(torch.equal(t.grad, w) for t, w in zip(leaves, want))
            out, leaves, _ = recorded(kind, dim, seq)  # and with a gradient that is expanded: strides of 0
            want = torch.autograd.grad(out.sum(), leaves, retain_graph=True)
            with compiled_autograd._enable(lambda gm: torch.compile(gm, backend="aot_eager", fullgraph=True, dynamic=dynamic)):
                out.sum().backward()
            assert all(torch.equal(t.grad, w) for t, w in zip(leaves, want))
    finally:
        set_backward("auto")
        torch._dynamo.reset()
