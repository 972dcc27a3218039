"""Rows of experts by their experts' matrices (csrc/gemm_pair.cu, grouped) against float64."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _unit(act, z, limit):
    if act in ("silu", "clamped"):
        g, u = z.chunk(2, dim=-1)
        if act == "silu":
            return torch.nn.functional.silu(g) * u
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1.0)
    return {None: lambda v: v, "relu2": lambda v: torch.relu(v).square(), "gelu": torch.nn.functional.gelu}[act](z)


# Rows per expert around a tile's 256 and the steps of 16 and 32 of its width, experts without rows, one expert, more
# experts than a warp counts at a time; features and k off the tiles' 256, 128 and 64.
@pytest.mark.parametrize("rows", [[1], [0, 31, 32, 33, 0, 0, 1], [255, 256, 257, 0, 513], [700], [16, 17, 300, 128, 129],
                                  [3, 0, 1] * 23, [1] * 512])
@pytest.mark.parametrize("n,k", [(256, 64), (64, 8), (40, 136), (600, 328)])
@pytest.mark.parametrize("act", [None, "relu2", "gelu", "silu", "clamped"])
def test_every_row_meets_its_experts_matrix(rows, n, k, act):
    from pulsarlm_b200.kernels import ops

    ops.require_device()
    gen = torch.Generator(device=DEV).manual_seed(sum(rows) + n + k)
    experts, total, limit = len(rows), sum(rows), 1.5
    x = torch.randn((total, k), generator=gen, device=DEV).bfloat16()
    w = (torch.randn((experts, 2 * n if act in ("silu", "clamped") else n, k), generator=gen, device=DEV) / k ** 0.5).bfloat16()
    ends = torch.tensor(rows, dtype=torch.int32, device=DEV).cumsum(0).int()
    out = torch.full((total + 1, n), 7.0, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.gemm_bf16_grouped(x, w, ends, out[:total], act, limit, status)
    got, first = out[:total].double(), 0
    for e, count in enumerate(rows):
        mine = slice(first, first + count)
        first += count
        if count == 0:
            continue
        z = x[mine].double() @ w[e].double().t()
        want = _unit(act, z, limit)
        # The product is off by one bfloat16 rounding (2^-9 of it), which the unit passes on with a slope of at most 2 |z| + 2 in
        # each factor, and the result by one more; the other factor of a gated unit is its own size.
        size = z.abs() if act not in ("silu", "clamped") else z.abs().reshape(count, 2, n).prod(1) + z.abs().reshape(count, 2, n).sum(1)
        bound = 2.0 ** -8 * ((2 * z.abs() + 2) * z.abs() if act in ("relu2", "gelu") else 2 * size) + 2.0 ** -8 * want.abs() + 1e-5
        assert bool(((got[mine] - want).abs() <= bound).all()), e
    assert int(status.item()) == 0 and bool((out[total] == 7.0).all())
