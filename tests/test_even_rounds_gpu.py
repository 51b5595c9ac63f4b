"""Batches just above what the warps of the GPU take at once, where the work is shared evenly instead of
leaving a few items to a round of their own."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu_delta, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 75])
@pytest.mark.parametrize("moves", [1185, 4440, 4441, 4500, 8881, 9000, 13321])
def test_deltas(n, moves, cuda):
    p, q = state.seeded_population(n, 7)
    cols = state.pq_to_columns(p, q)
    g = np.random.default_rng(moves)
    mv = np.stack((g.integers(0, 7, moves), g.integers(0, 2 * n, moves), g.integers(0, 2 * n, moves)), 1)
    mv = mv.astype(np.int32)
    dE, bad = gpu_delta.swap_deltas(cols, mv, badness=True)
    want, want_bad = gpu_delta.swap_deltas(cols, mv, badness=True, pairs=True)
    assert np.array_equal(dE, want) and np.array_equal(bad, want_bad)
