"""The weighted sum of branches four elements at a time gives the bits of the one-by-one form, whatever the partial sums."""

from __future__ import annotations

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,width", [(1, 4), (3, 36), (9, 2048), (5, 37)])  # the last: no whole quads
@pytest.mark.parametrize("splits", [(1,), (1, 1), (8, 3), (9, 1), (2, 1, 8, 5)])  # nine: more than are fetched together
def test_branch_sum(tokens, width, splits):
    from mini_engine_b200.csrc import ops

    torch.manual_seed(width + len(splits))
    branches = [(torch.randn(s, tokens, width, device="cuda"), 0.3 + 0.2 * i) for i, s in enumerate(splits)]
    out = torch.full((tokens, width), float("nan"), device="cuda")
    ops.branch_sum(branches, out)
    want = torch.zeros(tokens, width, dtype=torch.float64, device="cuda")
    for partial, factor in branches:
        whole = torch.zeros(tokens, width, device="cuda")
        for s in partial:
            whole = whole + s
        # one rounding of factor * whole + sum: exact in float64, then rounded
        want = (want.float().double() + torch.tensor(factor, dtype=torch.float32).double().item() * whole.double()).float().double()
    assert torch.equal(out, want.float())
