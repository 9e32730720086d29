"""The memory-bound helper kernels at the edges of their tiles: mask packing and the backward's statistics,
each against plain torch on the same inputs."""

import ctypes

import pytest
import torch

from kohakufa_b200 import _lib, op
from kohakufa_b200.mask import pack_mask_op

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


@pytest.mark.parametrize("dim", [16, 48, 64, 80, 128])
@pytest.mark.parametrize("seq", [1, 15, 17, 127, 128, 130])
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
