"""Delta rules in bfloat16: portions sixteen tokens a step of the scan beside the walk token by token, and steps of single
tokens, all against float64 on the same inputs."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _ops():
    from pulsarlm_b200.kernels import ops

    ops.require_device()
    return ops


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# Portions shorter than a chunk, of whole chunks, one more and one less, one past the pass of 128 chunks, singles between.
# Steps of single tokens have a form of their own (the last two; an entry may bring none or two).
LENGTHS = [[33], [1, 48, 1, 17, 15], [16, 0, 31], [2081], [5] * 12, [1] * 7, [2, 0, 1]]


def _both(ops, monkeypatch, name, call):
    """The call's (out, state) in chunks and token by token."""
    chunks = call()
    with monkeypatch.context() as m:
        m.setattr(ops.library(), name, lambda *a: 0)
        return chunks, call()


def _check(chunks, walk, want_out, want_state):
    for mine, theirs, want, bar in ((chunks[1], walk[1], want_state, 1e-6), (chunks[0], walk[0], want_out, 3e-3)):
        # (float32 sums of a few hundred terms of a state's memory; outputs are rounded to bfloat16 once, 2^-9 at most)
        assert _rel(mine, want) <= max(bar, 1.2 * _rel(theirs, want)), (_rel(mine, want), _rel(theirs, want))


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("heads,qk_heads,dim,vdim", [(3, 3, 64, 64), (4, 2, 32, 48), (2, 1, 128, 128), (2, 2, 64, 16)])
@pytest.mark.parametrize("rate", [-2.0, 1.0, 4.0])   # memories of many tokens, of a few, of none (decays that underflow)
def test_channel_decay_in_chunks(monkeypatch, lengths, heads, qk_heads, dim, vdim, rate):
    ops = _ops()
    gen = torch.Generator(device=DEV).manual_seed(dim + vdim + len(lengths))
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    tokens, n = sum(lengths), len(lengths)
    width = 2 * qk_heads * dim + heads * vdim
    proj = rand(tokens, width + heads + 3).to(BF)            # (rows that start on no 16 bytes)
    q, k = proj[:, :qk_heads * dim], proj[:, qk_heads * dim:2 * qk_heads * dim]
    v, b_pre = proj[:, 2 * qk_heads * dim:width], proj[:, width:width + heads]
    a_pre, gate = rand(tokens, heads * dim).to(BF) * 2, rand(tokens, heads * vdim).to(BF)
    a_log, dt_bias, norm = rate + 0.3 * rand(heads), rand(heads * dim) - 2, 1 + 0.1 * rand(vdim)
    start = 0.3 * rand(n + 2, heads, dim, vdim)
    slots = [n + 1 - i for i in range(n)]
    first = [sum(lengths[:i]) for i in range(n)]

    def call():
        state, out = start.clone(), torch.empty((tokens, heads * vdim), dtype=BF, device=DEV)
        ops.gated_delta(q, k, v, b_pre, a_pre, gate, a_log, dt_bias, norm, state, _i32(first), _i32(lengths), _i32(slots),
                        out, heads, qk_heads, dim, vdim, 1e-6, dim ** -0.5, 1e-5)
        return out, state

    chunks, walk = _both(ops, monkeypatch, "pl_gated_delta_chunk_floats", call)
    unit = lambda x: x.double().view(tokens, qk_heads, dim).repeat_interleave(heads // qk_heads, 1)  # noqa: E731
    qd, kd, vd = unit(q), unit(k), v.double().view(tokens, heads, vdim)
    qd = qd / (qd.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt() * dim ** -0.5
    kd = kd / (kd.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    g = torch.exp(-a_log.double().exp()[None, :, None]
                  * torch.nn.functional.softplus(a_pre.double() + dt_bias.double()).view(tokens, heads, dim))
    b = torch.sigmoid(b_pre.double())
    want = start.double()
    o = torch.empty((tokens, heads, vdim), dtype=torch.float64, device=DEV)
    for e in range(n):
        S = want[slots[e]]
        for t in range(first[e], first[e] + lengths[e]):
            S = S * g[t][..., None]
            u = b[t][:, None] * (vd[t] - torch.einsum("hij,hi->hj", S, kd[t]))
            S = S + kd[t][..., None] * u[:, None]
            o[t] = torch.einsum("hij,hi->hj", S, qd[t])
        want[slots[e]] = S
    o = o / (o.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * norm.double()
    _check(chunks, walk, o.reshape(tokens, -1) * torch.sigmoid(gate.double()), want)


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("heads,dim", [(3, 64), (4, 32), (2, 128)])
@pytest.mark.parametrize("scale", [math.exp(-0.5), 30.0])
def test_general_rule_in_chunks(monkeypatch, lengths, heads, dim, scale):
    ops = _ops()
    gen = torch.Generator(device=DEV).manual_seed(dim + len(lengths))
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    tokens, n, width = sum(lengths), len(lengths), heads * dim
    proj = rand(tokens, 5 * width + 1).to(BF)
    r, k, v, g, a = (proj[:, i * width:(i + 1) * width] for i in range(5))
    w_pre = rand(tokens, width).to(BF)
    w0, a0, norm = rand(width) - 3, rand(width), 1 + 0.1 * rand(width)
    start = 0.3 * rand(n + 2, heads, dim, dim)
    slots = [n + 1 - i for i in range(n)]
    first = [sum(lengths[:i]) for i in range(n)]

    def call():
        state, out = start.clone(), torch.empty((tokens, width), dtype=BF, device=DEV)
        ops.delta_rule(r, k, v, g, a, w_pre, w0, a0, norm, state, _i32(first), _i32(lengths), _i32(slots), out, heads, dim,
                       scale, 1e-6, 1e-5)
        return out, state

    chunks, walk = _both(ops, monkeypatch, "pl_delta_rule_chunk_floats", call)
    view = lambda x: x.double().view(tokens, heads, dim)  # noqa: E731
    u = view(k) / (view(k).pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    decay = torch.exp(-scale * torch.sigmoid(w_pre.double() + w0.double())).view(tokens, heads, dim)
    gone = torch.sigmoid(a.double() + a0.double()).view(tokens, heads, dim) * u
    want = start.double()
    o = torch.empty((tokens, heads, dim), dtype=torch.float64, device=DEV)
    for e in range(n):
        S = want[slots[e]]
        for t in range(first[e], first[e] + lengths[e]):
            read = torch.einsum("hij,hi->hj", S, u[t])
            S = decay[t][..., None] * S - gone[t][..., None] * read[:, None] + view(k)[t][..., None] * view(v)[t][:, None]
            o[t] = torch.einsum("hij,hi->hj", S, view(r)[t])
        want[slots[e]] = S
    o = (o / (o.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(tokens, -1) * norm.double()
    _check(chunks, walk, o * torch.sigmoid(g.double()), want)
