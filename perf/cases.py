"""The work whose speed is tracked: attention calls as programs make them, over the range of sizes they make
them at. ``listed()`` are fixed cases, ``draw()`` makes more of the same ranges; ``prepare`` / ``run`` / ``work`` /
``tolerance`` / ``exact`` say what one pass is, what it cannot do without and what its results have to be.

A case is a dict of plain values:
    kind      "plain" (dense, causal, block-causal), "mask" (a boolean mask given to the call) or "varlen"
    batch, heads, kv_heads, s_q, s_kv, dim, dtype, block (0 dense, 1 causal, P frames of P tokens)
    backward  True: forward + backward with the gradients of q, k, v; False: forward only, no autograd
    varlen: batch sequences, lengths 1 .. s_q drawn from ``length_seed``
    mask: a sliding window of ``window`` keys on either side, as a bool ``[1, 1, Sq, Skv]`` tensor
"""

import math
import random

import torch

from kohakufa_b200 import attention, attention_varlen, varlen_plan
from kohakufa_b200.workloads import visible_pairs

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _case(name, kind, batch, heads, s_q, dim, dtype, block=0, s_kv=None, kv_heads=None, backward=True, **more):
    case = dict(kind=kind, batch=batch, heads=heads, kv_heads=kv_heads or heads, s_q=s_q, s_kv=s_kv or s_q, dim=dim,
                dtype=dtype, block=block, backward=backward, **more)  # fmt: skip
    return dict(name=name, **case) if name else case


def listed():
    return [
        # one latency-bound inference call: a short prompt, few heads, no gradients
        _case("tiny_forward", "plain", 1, 8, 64, 64, "fp16", backward=False),
        # a small layer's training step: 2 x 512 tokens, launches and host time count
        _case("small_step", "plain", 2, 4, 512, 64, "fp16"),
        # vision transformer layer: many short sequences of 201 tokens (196 patches and 5 more)
        _case("vit_step", "plain", 32, 12, 201, 64, "fp16"),
        # image generation, cross attention of a latent grid to a short text; a head dim that is padded
        _case("cross_step", "plain", 4, 8, 4096, 40, "fp16", s_kv=77),
        # language model prompt: causal, grouped queries, forward only
        _case("gqa_prefill", "plain", 1, 32, 4096, 128, "bf16", block=1, kv_heads=8, backward=False),
        # video: frames of 256 tokens, each sees itself and the earlier ones
        _case("video_step", "plain", 8, 16, 4096, 64, "fp16", block=256),
        # dense self attention of a length that is no multiple of any tile
        _case("dense_ragged_step", "plain", 2, 16, 4100, 64, "fp16"),
        # dense self attention at head dim 128
        _case("dense_wide_step", "plain", 1, 16, 4096, 128, "fp16"),
        # a head dim between the common ones, causal
        _case("dim96_step", "plain", 2, 16, 2048, 96, "bf16", block=1),
        # sliding-window attention through a boolean mask that the call packs
        _case("window_mask_step", "mask", 1, 16, 2048, 64, "bf16", window=256),
        # packed documents of different lengths, causal, grouped queries
        _case("packed_step", "varlen", 16, 16, 2048, 128, "bf16", block=1, kv_heads=4, length_seed=7),
        # long-context language model training: 2 x 8192 tokens, 32 heads
        _case("long_causal_step", "plain", 2, 32, 8192, 128, "bf16", block=1),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    most = 0.8 * work(listed()[-1])["flops"]
    while True:
        kind = rng.choice(["plain"] * 6 + ["mask", "varlen"])
        dtype = rng.choice(["fp16", "bf16"])
        dim = rng.choice([64] * 5 + [128] * 5 + [96, 80, 32, 40, 72])
        heads = rng.choice([4, 8, 12, 16, 32])
        kv_heads = heads // rng.choice([1, 1, 2, 4])
        batch = _log_uniform(rng, 1, 32)
        block = rng.choice([0, 0, 1, 1, _log_uniform(rng, 16, 512)])
        backward = rng.random() < 0.75
        if kind == "mask":
            s = _log_uniform(rng, 128, 4096)
            case = _case(None, kind, min(batch, 4), heads, s, dim, dtype, 0, None, kv_heads, backward, window=_log_uniform(rng, 16, s))
        elif kind == "varlen":
            dim = 16 * -(-dim // 16)
            s = _log_uniform(rng, 64, 4096)
            case = _case(None, kind, batch, heads, s, dim, dtype, block, None, kv_heads, backward, length_seed=rng.randrange(1000))
        else:
            s = _log_uniform(rng, 48, 8192)
            s_kv = _log_uniform(rng, 48, 4096) if block == 0 and rng.random() < 0.25 else s
            case = _case(None, kind, batch, heads, s, dim, dtype, block, s_kv, kv_heads, backward)
        rows = case["batch"] * max(case["s_q"], case["s_kv"]) * heads
        if work(case)["flops"] <= most and rows * dim <= 2 * 32 * 8192 * 128:
            return case


def _lengths(case):
    rng = random.Random(case["length_seed"])
    lengths = [rng.randint(1, case["s_q"]) for _ in range(case["batch"])]
    lengths[0] = case["s_q"]
    return lengths


def _inputs(case, seed):
    """q, k, v, dout: normal values (of 0.5 at head dim 128, where the scores are then of the usual size),
    as projections lay them out: [B, S, H, D] storage viewed as [B, H, S, D], or packed [T, H, D]."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    std = 0.5 if case["dim"] == 128 else 1.0

    def one(rows, heads):
        x = torch.randn(*rows, heads, case["dim"], generator=gen, device="cuda") * std
        return x.to(DTYPES[case["dtype"]])

    if case["kind"] == "varlen":
        total = sum(_lengths(case))
        return tuple(one((total,), h) for h in (case["heads"], case["kv_heads"], case["kv_heads"], case["heads"]))
    b = case["batch"]
    q, k, v, dout = (
        one((b, s), h)
        for s, h in ((case["s_q"], case["heads"]), (case["s_kv"], case["kv_heads"]), (case["s_kv"], case["kv_heads"]), (case["s_q"], case["heads"]))
    )
    return tuple(t.transpose(1, 2) for t in (q, k, v, dout))


def _window_mask(case):
    rows = torch.arange(case["s_q"], device="cuda")[:, None]
    cols = torch.arange(case["s_kv"], device="cuda")[None, :]
    return ((rows - cols).abs() <= case["window"])[None, None]


def prepare(case, seed):
    q, k, v, dout = _inputs(case, seed)
    state = {"case": case, "dout": dout}
    state["qkv"] = tuple(t.requires_grad_() if case["backward"] else t for t in (q, k, v))
    if case["kind"] == "mask":
        state["mask"] = _window_mask(case)
    if case["kind"] == "varlen":
        ends = torch.tensor([0] + _lengths(case)).cumsum(0)
        state["cu"] = ends.to(torch.int32).cuda()
        state["plan"] = varlen_plan(state["cu"], state["cu"])
    return state


def _forward(state):
    case = state["case"]
    q, k, v = state["qkv"]
    if case["kind"] == "varlen":
        return attention_varlen(q, k, v, state["cu"], state["cu"], block_causal=case["block"], plan=state["plan"])
    if case["kind"] == "mask":
        return attention(q, k, v, mask=state["mask"])
    if case["block"] == 1:
        return attention(q, k, v, causal=True)
    return attention(q, k, v, block_causal=case["block"])


def run(state):
    if not state["case"]["backward"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    return (out.detach(), *torch.autograd.grad(out, state["qkv"], state["dout"]))


def _pairs(case):
    """Visible (query, key) pairs of one head, over the whole batch."""
    if case["kind"] == "varlen":
        return sum(visible_pairs(n, n, case["block"]) for n in _lengths(case))
    if case["kind"] == "mask":
        s_kv, w = case["s_kv"], case["window"]
        return case["batch"] * sum(max(0, min(s_kv, r + w + 1) - max(0, r - w)) for r in range(case["s_q"]))
    return case["batch"] * visible_pairs(case["s_q"], case["s_kv"], case["block"])


def work(case):
    """Two matrix products of the visible pairs forward, five more backward; q, k, v (and dout) read once, the
    output (and three gradients) written once, the mask read once."""
    flops = 4.0 * case["heads"] * case["dim"] * _pairs(case) * (3.5 if case["backward"] else 1.0)
    if case["kind"] == "varlen":
        rows_q = rows_kv = sum(_lengths(case))
    else:
        rows_q, rows_kv = case["batch"] * case["s_q"], case["batch"] * case["s_kv"]
    q_bytes, kv_bytes = (2 * case["dim"] * h * r for h, r in ((case["heads"], rows_q), (case["kv_heads"], rows_kv)))
    moved = 2 * q_bytes + 2 * kv_bytes  # q, out, k, v
    if case["backward"]:
        moved += 2 * q_bytes + 2 * kv_bytes  # dout, dq, dk, dv
    if case["kind"] == "mask":
        moved += case["s_q"] * case["s_kv"]
    return {"bytes": float(moved), "flops": flops}


def tolerance(case):
    """About four times the distance of the kernels from fp64 on these inputs: 3e-4 in fp16 and 2.4e-3 in bf16 (P and dS
    are rounded to 16 bits before the second product, outputs and gradients once more)."""
    return {"rel": 1.2e-3 if case["dtype"] == "fp16" else 1e-2}


def _exact_head(q, k, v, dout, visible, scale):
    """fp64 attention of one query head: out, dq, dk, dv (the last three None without dout)."""
    s = (q @ k.T).mul_(scale)
    if visible is not None:
        s.masked_fill_(~visible, float("-inf"))
    p = torch.softmax(s, -1)
    out = p @ v
    if dout is None:
        return out, None, None, None
    dv = p.T @ dout
    ds = (dout @ v.T).sub_((dout * out).sum(-1, keepdim=True)).mul_(p)
    return out, (ds @ k).mul_(scale), (ds.T @ q).mul_(scale), dv


def _exact_sequence(case, q, k, v, dout, visible):
    """[H, S, D] inputs of one sequence; results in fp64."""
    group = case["heads"] // case["kv_heads"]
    scale = case["dim"] ** -0.5
    out, dq = torch.zeros_like(q, dtype=torch.float64), torch.zeros_like(q, dtype=torch.float64)
    dk, dv = torch.zeros_like(k, dtype=torch.float64), torch.zeros_like(v, dtype=torch.float64)
    for h in range(case["heads"]):
        g = dout[h].double() if case["backward"] else None
        o, a, b, c = _exact_head(q[h].double(), k[h // group].double(), v[h // group].double(), g, visible, scale)
        out[h] = o
        if case["backward"]:
            dq[h] = a
            dk[h // group] += b
            dv[h // group] += c
    return (out, dq, dk, dv) if case["backward"] else (out,)


def _visible(case, s_q, s_kv):
    if case["kind"] == "mask":
        return _window_mask(case)[0, 0]
    if case["block"] == 0:
        return None
    rows = torch.arange(s_q, device="cuda")[:, None] // case["block"]
    cols = torch.arange(s_kv, device="cuda")[None, :] // case["block"]
    return cols <= rows


@torch.no_grad()
def exact(case, seed):
    q, k, v, dout = _inputs(case, seed)
    if case["kind"] == "varlen":
        parts, start = [], 0
        for n in _lengths(case):
            q1, k1, v1, d1 = (t[start : start + n].transpose(0, 1) for t in (q, k, v, dout))
            parts.append([t.transpose(0, 1) for t in _exact_sequence(case, q1, k1, v1, d1, _visible(case, n, n))])
            start += n
        results = tuple(torch.cat(ts) for ts in zip(*parts))
    else:
        visible = _visible(case, case["s_q"], case["s_kv"])
        parts = [_exact_sequence(case, q[b], k[b], v[b], dout[b], visible) for b in range(case["batch"])]
        results = tuple(torch.stack(ts) for ts in zip(*parts))
    return results if case["backward"] else results[0]
