"""Which (batch, head, tile) a CTA works on and which keys a row sees, where the divisions behind them have remainders."""

import ctypes

import pytest
import torch

from kohakufa_b200 import _lib, attention, op, set_backward
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


@pytest.mark.parametrize("dim", [48, 64, 128])
def test_both_kinds_of_backward_ctas_in_one_launch(dim):
    """dK, dV and dQ of one launch are those of a launch each, bit for bit."""
    gen = torch.Generator().manual_seed(dim)
    q, k, v, dout = (torch.randn(2, 300, 3, dim, generator=gen).half().cuda().transpose(1, 2) for _ in range(4))
    out, lse = op.attention_fwd_op(q, k, v, 0.125, 1)
    set_backward("split")
    try:
        want = op.attention_bwd_op(q, k, v, out, dout, lse, 0.125, 1)
    finally:
        set_backward("auto")
    got = [torch.full_like(t, 7.0) for t in want]
    lib, ref = _lib.load(), lambda t: ctypes.byref(_lib.tensor4(t))
    stats = torch.empty(lib.kfa_bwd_stats_bytes(2, 3, 300) // 4, device="cuda")
    word, stream, code = _lib.status_word(q.device).data_ptr(), _lib.stream_ptr(q.device), _lib.dtype_code(q.dtype)
    qkvg = [ref(t) for t in (q, k, v, dout)]
    assert lib.kfa_bwd_prepare(ref(out), ref(dout), lse.data_ptr(), stats.data_ptr(), code, stream) == 0
    assert lib.kfa_bwd_dkdv(*qkvg, stats.data_ptr(), ref(got[1]), ref(got[2]), 0.125, 1, code, word, stream) == 0
    assert lib.kfa_bwd_dq(*qkvg, stats.data_ptr(), ref(got[0]), 0.125, 1, code, word, stream) == 0
    assert all(torch.equal(a, b) for a, b in zip(got, want))
