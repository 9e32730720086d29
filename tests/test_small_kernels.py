"""The memory-bound helper kernels at the edges of their tiles: mask packing and the backward's statistics,
each against plain torch on the same inputs."""

import ctypes

import pytest
import torch

from kohakufa_b200 import _lib, attention, op, set_backward
from kohakufa_b200.mask import pack_mask_op
from oracle import reference as oracle

pytestmark = pytest.mark.gpu


def unpack(words, n):
    """Bits of ``words [..., ceil(n / 128) * 4]`` as bool, and that the padding is clear."""
    flat = ((words.unsqueeze(-1) >> torch.arange(32, device=words.device)) & 1).flatten(-2).bool()
    assert not bool(flat[..., n:].any())
    return flat[..., :n]


@pytest.mark.parametrize("s_q,s_kv", [(1, 1), (31, 33), (32, 128), (127, 129), (129, 1), (160, 96), (257, 384)])
@pytest.mark.parametrize("layout", ["plain", "transposed", "expanded", "sliced"])
def test_pack_mask_edges(s_q, s_kv, layout):
    """Whole numbers: equal, not close."""
    gen = torch.Generator().manual_seed(s_q * 1000 + s_kv)
    if layout == "transposed":
        mask = (torch.rand(2, 1, s_kv, s_q, generator=gen) < 0.3).cuda().transpose(-1, -2)
    elif layout == "expanded":  # one row of visible keys for every query
        mask = (torch.rand(1, 2, 1, s_kv, generator=gen) < 0.3).cuda().expand(1, 2, s_q, s_kv)
    elif layout == "sliced":
        mask = (torch.rand(1, 2, s_q + 3, 2 * s_kv + 1, generator=gen) < 0.3).cuda()[:, :, 3:, 1::2]
    else:
        mask = (torch.rand(2, 2, s_q, s_kv, generator=gen) < 0.01).cuda()
    words, words_t, tiles = pack_mask_op(mask, s_q, s_kv)
    assert torch.equal(unpack(words, s_kv), mask)
    assert torch.equal(unpack(words_t, s_q), mask.transpose(-1, -2))
    padded = torch.nn.functional.pad(mask, (0, -s_kv % 128, 0, -s_q % 128))
    want = padded.unflatten(-1, (-1, 128)).unflatten(-3, (-1, 128)).any(-1).any(-2)
    assert torch.equal(tiles != 0, want)


@pytest.mark.parametrize("dim", [16, 32, 48, 64, 80, 112, 128])
@pytest.mark.parametrize("seq", [1, 15, 17, 65, 127, 128, 130])
def test_backward_statistics(dim, seq):
    """(-m, -log2 l, -delta) per row, padded rows (-inf, 0, 0). delta is a sum of ``dim`` fp32 products: its
    error is at most dim * 2^-24 of the sum of the products' magnitudes in either order of summation."""
    gen = torch.Generator().manual_seed(dim + seq)
    out, dout = (torch.randn(2, seq, 3, dim, generator=gen).bfloat16().cuda().transpose(1, 2) for _ in range(2))
    lse = torch.randn(2, 3, 2, seq, generator=gen).cuda()
    lib = _lib.load()
    tiles = -(-seq // 128)
    stats = torch.full((2, 3, tiles, 3, 128), 7.0, device="cuda")
    acc = torch.full((2 * 3 * tiles * 128 * dim,), 7.0, device="cuda") if dim in op.FUSED_DIMS else None
    args = [ctypes.byref(_lib.tensor4(out)), ctypes.byref(_lib.tensor4(dout)), lse.data_ptr(), stats.data_ptr()]
    tail = [_lib.KFA_BF16, _lib.stream_ptr(out.device)]
    _lib.check(lib.kfa_bwd_prepare(*args, *tail))
    plain = stats.clone()
    if acc is not None:
        stats.fill_(7.0)
        _lib.check(lib.kfa_bwd_prepare_fused(*args, acc.data_ptr(), *tail))
        assert torch.equal(stats, plain) and not bool(acc.any())
    rows = plain.permute(0, 1, 3, 2, 4).flatten(-2)  # [B, H, 3, padded rows]
    assert torch.equal(rows[:, :, :2, :seq], -lse)
    products = out.double() * dout.double()
    error = (rows[:, :, 2, :seq].double() + products.sum(-1)).abs()
    assert bool((error <= dim * 2.0**-24 * products.abs().sum(-1)).all())
    assert bool((rows[:, :, 0, seq:] == -torch.inf).all()) and not bool(rows[:, :, 1:, seq:].any())


@pytest.mark.parametrize("dim,dtype", [(40, torch.float16), (64, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("s_q,s_kv,heads,kv_heads,block", [(4096, 77, 4, 4, 0), (1025, 128, 4, 2, 0), (2000, 129, 2, 1, 0), (2100, 200, 2, 2, 1), (3100, 300, 2, 1, 100)])
def test_shared_out_steps(dim, dtype, s_q, s_kv, heads, kv_heads, block):
    """Few key tiles: several CTAs share a tile's steps and their fp32 parts are summed. dQ is the split kernels' own;
    dK, dV differ from theirs by the order of fp32 sums, then one rounding to 16 bits (a unit in the last place: 2^-10,
    2^-7 of a value), and repeat bit for bit."""
    gen = torch.Generator().manual_seed(s_q + s_kv)

    def one(seq, h):
        return torch.randn(1, seq, h, dim, generator=gen).to(dtype).cuda().transpose(1, 2)

    q, k, v, dout = one(s_q, heads), one(s_kv, kv_heads), one(s_kv, kv_heads), one(s_q, heads)
    lib, host, word = _lib.load(), _lib.host(), _lib.status_word(q.device)
    ref = lambda t: ctypes.byref(_lib.tensor4(t))  # noqa: E731
    assert lib.kfa_bwd_parts_bytes(ref(q), ref(k)) > 0
    out, lse = host.forward(q, k, v, dim**-0.5, block, word)
    got = host.backward(q, k, v, out, dout, lse, dim**-0.5, block, word, 0)
    again = host.backward(q, k, v, out, dout, lse, dim**-0.5, block, word, 2)
    assert all(torch.equal(a, b) for a, b in zip(got, again))
    like = lambda t: torch.empty_like(t.transpose(1, 2).contiguous()).transpose(1, 2)  # noqa: E731
    want = [like(t) for t in (q, k, v)]
    stats = torch.empty(lib.kfa_bwd_stats_bytes(1, heads, s_q) // 4, device="cuda")
    _lib.check(lib.kfa_bwd_narrow(*(ref(t) for t in (q, k, v, out, dout)), lse.data_ptr(), stats.data_ptr(), None,
                                  *(ref(t) for t in want), dim**-0.5, block, _lib.dtype_code(dtype), word.data_ptr(),
                                  _lib.stream_ptr(q.device)))  # fmt: skip
    assert _lib.device_status() == 0 and torch.equal(got[0], want[0])
    ulp = 2.0**-10 if dtype == torch.float16 else 2.0**-7
    for a, b in zip(got[1:], want[1:]):
        a, b = a.double(), b.double()
        # the fp32 sums: at most the count of summed products (queries x heads of the group) times 2^-24 of the largest sum
        noise = s_q * (heads // kv_heads) * 2.0**-24 * float(b.abs().max())
        assert bool(((a - b).abs() <= ulp * b.abs() + noise + 2.0**-24).all())


@pytest.mark.parametrize("dim", [40, 64, 128])
def test_shared_out_steps_of_a_batch(dim):
    """Several batch entries and grouped heads on the shared-out route, through the public call and against fp64 (tolerance of
    the other fp16 parity tests: P, dS and the results are rounded to 11 bits)."""
    gen = torch.Generator().manual_seed(dim)
    q, k, v, dout = (torch.randn(3, s, h, dim, generator=gen).half().cuda().transpose(1, 2) for s, h in ((1100, 4), (77, 2), (77, 2), (1100, 4)))
    ref = lambda t: ctypes.byref(_lib.tensor4(t))  # noqa: E731
    assert _lib.load().kfa_bwd_parts_count(ref(q), ref(k), int(dim == 64)) == 4
    qkv = [t.requires_grad_() for t in (q, k, v)]
    out = attention(*qkv)
    got = (out, *torch.autograd.grad(out, qkv, dout))
    assert _lib.device_status() == 0
    for g, w in zip(got, oracle.attention_fp64(q, k, v, dout, dim**-0.5, groups=2)):
        assert oracle.metrics(g, w)["rel_err"] < 5e-3


@pytest.mark.parametrize("dim", [64, 80])
def test_split_mode_does_not_depend_on_the_batch(dim):
    """In "split" mode a batch entry's gradients are the bits of that entry alone, also where queries outnumber keys so far
    that "auto" shares out a key tile's steps by the number of tiles in the batch."""
    gen = torch.Generator().manual_seed(dim)
    q, k, v, dout = (torch.randn(3, s, 2, dim, generator=gen).half().cuda().transpose(1, 2) for s in (2100, 77, 77, 2100))

    def grads(rows):
        qkv = [t[rows].detach().requires_grad_() for t in (q, k, v)]
        return torch.autograd.grad(attention(*qkv), qkv, dout[rows])

    try:
        set_backward("split")
        whole, alone = grads(slice(0, 3)), grads(slice(1, 2))
    finally:
        set_backward("auto")
    assert all(torch.equal(a[1:2], b) for a, b in zip(whole, alone))
