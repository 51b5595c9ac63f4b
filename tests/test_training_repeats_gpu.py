"""Training on batches of up to 256 rows gives the same bits every time: no gradient is added up from more than two
parts whose order could change."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import learned, state, tempering

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [64, 100, 128, 129, 200, 256])
def test_same_bits(batch, cuda):
    p, q = state.seeded_population(40, 16)
    cols = state.pq_to_columns(p, q)
    runs = []
    for _ in range(5):
        ch = tempering.TemperingChains(cols, np.geomspace(0.05, 5.0, 16), 5, ladder_size=16)
        lp = learned.LearnedProposal(ch, seed=2, ring_capacity=1 << 14, moves=16, batch=batch)
        for _ in range(4):
            lp.step()
        for _ in range(12):
            lp.train()
        runs.append((lp.params.cpu().numpy(), lp.grads.cpu().numpy(), lp.adam_v.cpu().numpy()))
    for run in runs[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(runs[0], run))
