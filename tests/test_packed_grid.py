"""Packed batches: the numbering of tiles without gaps, the rectangular one, and the rows no sequence owns."""

import ctypes

import pytest
import torch

from kohakufa_b200 import _lib, attention_varlen, op, varlen_plan

pytestmark = pytest.mark.gpu


def run(q, k, v, dout, cu, plan, **kw):
    qkv = [t.detach().requires_grad_() for t in (q, k, v)]
    out = attention_varlen(*qkv, cu, cu, plan=plan, **kw)
    grads = torch.autograd.grad(out, qkv, dout)
    assert _lib.device_status() == 0
    return [out.detach(), *grads]


def packed(lengths, heads, kv_heads, dim, extra=0):
    gen = torch.Generator().manual_seed(len(lengths))
    total = sum(lengths) + extra
    ts = [torch.randn(total, h, dim, generator=gen).bfloat16().cuda() for h in (heads, kv_heads, kv_heads, heads)]
    return *ts, torch.tensor([0, *lengths]).cumsum(0).int().cuda()


@pytest.mark.parametrize("n_seqs,longest", [(1, 1), (31, 300), (33, 700), (256, 90), (257, 90), (300, 400)])
@pytest.mark.parametrize("causal", [True, False])
def test_batch_equals_its_halves(n_seqs, longest, causal):
    """A sequence's results do not depend on the batch it is in, so a batch equals its two halves bit for bit."""
    gen = torch.Generator().manual_seed(longest)
    lengths = torch.randint(0, longest + 1, (n_seqs,), generator=gen).tolist()
    lengths[n_seqs // 2] = longest
    check_halves(lengths, causal)


@pytest.mark.parametrize("n_seqs,others", [(40, 130), (600, 40)])
@pytest.mark.parametrize("causal", [True, False])
def test_one_long_sequence(n_seqs, others, causal):
    """Most of the rectangle's tiles do not exist: numbered without gaps (40 sequences: two scans of 32 lengths, 600:
    nineteen); the half of the 600 that the long one is not in has one tile a sequence and is a rectangle."""
    gen = torch.Generator().manual_seed(n_seqs)
    lengths = torch.randint(1, others + 1, (n_seqs,), generator=gen).tolist()
    lengths[-2] = 2900
    check_halves(lengths, causal)


def check_halves(lengths, causal):
    n_seqs = len(lengths)
    q, k, v, dout, cu = packed(lengths, 4, 2, 64)
    whole = run(q, k, v, dout, cu, varlen_plan(cu, cu), causal=causal)
    cut = (n_seqs + 1) // 2
    parts = []
    for a, b in ((0, cut), (cut, n_seqs)):
        if a == b or sum(lengths[a:b]) == 0:
            continue
        rows = slice(int(cu[a]), int(cu[b]))
        sub = (cu[a : b + 1] - cu[a]).contiguous()
        parts.append(run(q[rows], k[rows], v[rows], dout[rows], sub, varlen_plan(sub, sub), causal=causal))
    for i, w in enumerate(whole):
        assert torch.equal(w, torch.cat([p[i] for p in parts]))


@pytest.mark.parametrize("n_seqs", [3, 300])
def test_rows_outside_the_sequences_are_zero(n_seqs):
    """Freed memory full of NaN is what fresh outputs come from; rows before and after the sequences still read as zero,
    and so do the statistics."""
    lengths = [200, 300, 129] + [2] * (n_seqs - 3)
    q, k, v, dout, cu = packed(lengths, 2, 2, 64, extra=40)
    cu = cu + 7
    total = q.shape[0]
    junk = [torch.full((total, 2, 64), float("nan"), dtype=q.dtype, device="cuda") for _ in range(8)]
    lse = [torch.full((1, 2, 2, total), float("nan"), device="cuda") for _ in range(2)]
    del junk, lse
    out, dq, dk, dv = run(q, k, v, dout, cu, varlen_plan(cu, cu), causal=True)
    rows = torch.arange(total, device="cuda")
    inside = (rows >= cu[0]) & (rows < cu[-1])
    for t in (out, dq, dk, dv):
        assert bool(torch.isfinite(t).all()) and not bool(t[~inside].any())
        assert float(t[inside].abs().flatten(1).sum(-1).gt(0).float().mean()) > 0.9
    direct = op.varlen_fwd_op(q, k, v, cu, cu, 300, 300, 64**-0.5, 1)
    assert torch.equal(direct[0], out) and not bool(direct[1][..., ~inside].any())


@pytest.mark.parametrize("heads,dim", [(1, 16), (3, 48), (5, 128)])
@pytest.mark.parametrize("first,tail", [(0, 1), (1, 63), (64, 64), (30, 300)])
def test_left_over_rows_of_any_width(heads, dim, first, tail):
    """Rows of 16 to 640 columns (a warp stores 256 at a time), left over in pieces that begin and end inside a CTA's 64;
    a tensor of padded rows keeps its padding."""
    lib, total = _lib.load(), first + 70 + tail
    cu = torch.tensor([first, first + 70], dtype=torch.int32, device="cuda")
    wide = torch.full((total, heads, dim + 8), 3.0, dtype=torch.bfloat16, device="cuda")
    out = wide[..., :dim]
    lse = torch.full((1, heads, 2, total), 3.0, device="cuda")
    _lib.check(lib.kfa_varlen_zero_rows(ctypes.byref(_lib.tensor4(op._as4(out))), 1, cu.data_ptr(), cu.data_ptr(), 1, 70, 70,
                                        lse.data_ptr(), _lib.stream_ptr(out.device)))  # fmt: skip
    left = torch.ones(total, dtype=torch.bool, device="cuda")
    left[first : first + 70] = False
    assert not bool(out[left].any()) and not bool(lse[..., left].any())
    assert bool((out[~left] == 3).all()) and bool((lse[..., ~left] == 3).all()) and bool((wide[..., dim:] == 3).all())


def test_plan_shorter_than_a_sequence():
    """Rows past the longest length that a hand-made plan states (in whole tiles) are not computed: zeros in every output,
    out of freed memory full of NaN, and the other sequence is as it is alone."""
    q, k, v, dout, cu = packed([600, 100], 4, 2, 64)
    junk = [torch.full((700, 4, 64), float("nan"), dtype=q.dtype, device="cuda") for _ in range(8)]
    stats = torch.full((1 << 20,), float("nan"), device="cuda")
    del junk, stats
    got = run(q, k, v, dout, cu, (2, 120, 120))
    sub = torch.tensor([0, 100], dtype=torch.int32, device="cuda")
    alone = run(*(t[600:] for t in (q, k, v, dout)), sub, (1, 100, 100))
    for t, one, covered in zip(got, alone, (256, 128, 128, 128)):  # query rows of a tile of the forward, of the backward, keys
        assert bool(torch.isfinite(t).all()) and not bool(t[covered:600].any())
        assert bool(t[:covered].any(-1).all()) and torch.equal(t[600:], one)
