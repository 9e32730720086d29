"""The ends of the kernels: output rows leave through shared memory, whole rows at a time, and a launch that finds an earlier
failure in the status word leaves NaN whatever its roles had already done."""

import pytest
import torch

from kohakufa_b200 import _lib, attention, reset_status, set_backward
from oracle import reference as oracle

pytestmark = pytest.mark.gpu


def problem(dim, s_q, s_kv, dtype):
    gen = torch.Generator().manual_seed(1000 * dim + s_q)
    mk = lambda s: torch.randn(2, s, 2, dim, generator=gen).to(dtype).cuda().transpose(1, 2)  # noqa: E731
    return [mk(s_q).requires_grad_(), mk(s_kv).requires_grad_(), mk(s_kv).requires_grad_()], mk(s_q)


# Rows: one, a warp less one and more one, a tile less one and more one, a CTA of the forward and one row. fp16 results: P, dS
# and the outputs are each rounded to 11 bits, 2^-11 = 4.9e-4 relative; a row in the wrong place is an error of order 1.
@pytest.mark.parametrize("mode", ["split", "fused"])
@pytest.mark.parametrize("s_q,s_kv", [(1, 33), (31, 129), (33, 1), (127, 257), (129, 31), (257, 127)])
@pytest.mark.parametrize("dim", [16, 24, 32, 40, 48, 64, 72, 80, 96, 104, 112, 128])
def test_rows_and_columns_of_the_outputs(dim, s_q, s_kv, mode):
    if mode == "fused" and dim not in (64, 128):
        pytest.skip("the fused backward is built for head dims 64 and 128")
    leaves, dout = problem(dim, s_q, s_kv, torch.float16)
    set_backward(mode)
    try:
        out = attention(*leaves)
        got = (out.detach(), *torch.autograd.grad(out, leaves, dout))
    finally:
        set_backward("auto")
    want = oracle.attention_fp64(*(t.detach() for t in leaves), dout, dim**-0.5)
    for g, w in zip(got, want):
        # (with one key dS is a difference of equal numbers: its gradients are rounding noise around zero)
        scale = max(float(w.double().norm()), 1e-2 * float(dout.double().norm()))
        assert float((g.double().cpu() - w.double().cpu()).norm()) < 5e-3 * scale


@pytest.mark.parametrize("kind,dim", [("split", 128), ("fused", 64), ("fused", 128), ("mask", 64), ("hidden", 64)])
def test_an_earlier_failure_leaves_nan(kind, dim):
    leaves, dout = problem(dim, 300, 200, torch.float16)
    mask = None
    if kind in ("mask", "hidden"):
        mask = torch.zeros(300, 200, dtype=torch.bool, device="cuda")
        mask[:, :100] = kind == "mask"
    set_backward(kind if kind in ("split", "fused") else "auto")
    try:
        out = attention(*leaves, mask=mask)
        _lib.status_word(dout.device).fill_(105)
        grads = torch.autograd.grad(out, leaves, dout)
        again = attention(*(t.detach() for t in leaves), mask=mask)
        torch.cuda.synchronize()
        assert _lib.device_status() == 105
        assert all(bool(torch.isnan(t).all()) for t in (*grads, again))
    finally:
        reset_status()
        set_backward("auto")
    assert bool(torch.isfinite(attention(*(t.detach() for t in leaves), mask=mask)).all())
