"""Embedding rows: four values a load where rows are whole pieces, one at a time elsewhere."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [4, 129, 1020, 1024, 4100])
@pytest.mark.parametrize("tokens", [1, 67])
def test_rows_are_the_tables_and_bad_ids_give_zeros(dtype, width, tokens):
    from pulsarlm_b200.kernels import ops

    ops.require_device()
    table = torch.randn((50, width), device=DEV).to(dtype)
    ids = torch.randint(0, 50, (tokens,), dtype=torch.int32, device=DEV)
    for scale in (1.0, 1.5):
        out, status = torch.full((tokens, width), 9.0, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        ops.embed(table, ids, out, status, scale)
        assert torch.equal(out, table[ids.long()].float() * scale) and int(status.item()) == 0
        wrong = ids.clone()
        wrong[-1] = 50
        ops.embed(table, wrong, out, status, scale)
        assert int(status.item()) == 1 and not bool(out[-1].any()) and torch.equal(out[:-1], table[ids[:-1].long()].float() * scale)
