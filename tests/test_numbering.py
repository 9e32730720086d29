"""Which (batch, head, tile) a CTA works on and which keys a row sees, where the divisions behind them have remainders."""

import pytest
import torch

from kohakufa_b200 import attention, set_backward
from oracle import reference as oracle

pytestmark = pytest.mark.gpu


# (batch x heads) pairs around the groups of 8 that the launch order has; frames of one token, around a tile, beyond the
# sequence. fp16: P, dS and the results are rounded to 11 bits each; a tile or a row in the wrong place is an error of order 1.
@pytest.mark.parametrize("mode", ["split", "fused"])
@pytest.mark.parametrize("batch,heads,kv_heads", [(1, 1, 1), (1, 7, 7), (3, 3, 1), (2, 8, 2), (1, 17, 17), (5, 6, 3)])
@pytest.mark.parametrize("frame", [0, 1, 3, 127, 128, 129, 100000])
def test_tiles_and_frames(batch, heads, kv_heads, frame, mode):
    gen = torch.Generator().manual_seed(heads + frame)
    mk = lambda h: torch.randn(batch, 300, h, 64, generator=gen).half().cuda().transpose(1, 2)  # noqa: E731
    leaves, dout = [mk(heads).requires_grad_(), mk(kv_heads).requires_grad_(), mk(kv_heads).requires_grad_()], mk(heads)
    set_backward(mode)
    try:
        out = attention(*leaves, block_causal=frame)
        got = (out.detach(), *torch.autograd.grad(out, leaves, dout))
    finally:
        set_backward("auto")
    want = oracle.attention_fp64(*(t.detach() for t in leaves), dout, 0.125, block=frame, groups=heads // kv_heads)
    for g, w in zip(got, want):
        assert oracle.metrics(g, w)["rel_err"] < 5e-3
