"""A launch that finds an earlier failure in the status word, on problems of many tiles: the producers stop in the middle of
their rings, with consumers waiting for copies that are not started, and every output is NaN."""

import pytest
import torch

from kohakufa_b200 import _lib, attention, attention_varlen, reset_status, ring, set_backward, varlen_plan
from oracle import reference as oracle

pytestmark = pytest.mark.gpu


def tensors(dim, s_q, s_kv, heads=2):
    gen = torch.Generator().manual_seed(dim + s_kv)
    return [torch.randn(1, s, heads, dim, generator=gen).half().cuda().transpose(1, 2) for s in (s_q, s_kv, s_kv, s_q)]


@pytest.fixture
def failed():
    word = _lib.status_word(torch.device("cuda", torch.cuda.current_device()))
    yield lambda: word.fill_(105)
    reset_status()
    set_backward("auto")


# (the parts of shared-out steps: 1100 queries x 77 keys in "auto" mode at a head dim without fused kernels)
@pytest.mark.parametrize("mode", ["split", "fused", "auto"])
@pytest.mark.parametrize("dim,s_q,s_kv", [(16, 1100, 1100), (40, 1100, 1100), (40, 1100, 77), (64, 1100, 1100), (64, 1100, 77), (128, 1100, 1100)])
def test_rings_stop(dim, s_q, s_kv, mode, failed):
    q, k, v, dout = tensors(dim, s_q, s_kv)
    leaves = [t.requires_grad_() for t in (q, k, v)]
    set_backward(mode)
    out = attention(*leaves)
    failed()
    grads = torch.autograd.grad(out, leaves, dout)
    again = attention(*(t.detach() for t in leaves))
    torch.cuda.synchronize()
    assert _lib.device_status() == 105
    assert all(bool(torch.isnan(t).all()) for t in (*grads, again))
    reset_status()
    out = attention(*leaves)
    got = (out.detach(), *torch.autograd.grad(out, leaves, dout))
    want = oracle.attention_fp64(*(t.detach() for t in leaves), dout, dim**-0.5)
    for g, w in zip(got, want):  # fp16: P, dS and the results are rounded to 11 bits each
        assert oracle.metrics(g, w)["rel_err"] < 5e-3


@pytest.mark.parametrize("dim", [64, 128])
def test_rings_of_packed_batches_stop(dim, failed):
    gen = torch.Generator().manual_seed(dim)
    q, k, v, dout = (torch.randn(1500, 2, dim, generator=gen).half().cuda() for _ in range(4))
    cu = torch.tensor([0, 1100, 1130, 1500], dtype=torch.int32, device="cuda")
    plan, leaves = varlen_plan(cu, cu), [t.requires_grad_() for t in (q, k, v)]
    out = attention_varlen(*leaves, cu, cu, plan=plan)
    failed()
    grads = torch.autograd.grad(out, leaves, dout)
    again = attention_varlen(*(t.detach() for t in leaves), cu, cu, plan=plan)
    torch.cuda.synchronize()
    assert all(bool(torch.isnan(t).all()) for t in (*grads, again))
    reset_status()
    assert bool(torch.isfinite(attention_varlen(*(t.detach() for t in leaves), cu, cu, plan=plan)).all())


def test_rings_of_context_parallel_steps_stop(failed):
    gen = torch.Generator().manual_seed(3)
    shards = [[torch.randn(1, 2048, 2, 128, generator=gen).half().cuda().transpose(1, 2) for _ in range(2)] for _ in range(4)]
    failed()
    outs, _, *grads = ring.emulate_ring(*shards)
    torch.cuda.synchronize()
    assert all(bool(torch.isnan(t).all()) for ts in (outs, *grads) for t in ts)
    reset_status()
    outs, _, *grads = ring.emulate_ring(*shards)
    assert all(bool(torch.isfinite(t).all()) for ts in (outs, *grads) for t in ts)
