"""Batched swap deltas around the edges of the slots a lane holds, and on states whose lines overflow the
small counters, against the literal pair formulation; few moves and many."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu_delta, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 16, 17, 32, 33, 48, 49, 64, 65, 75])
@pytest.mark.parametrize("moves", [1, 300, 5000])
def test_deltas_match_pairs(n, moves, cuda):
    p, q = state.seeded_population(n, 3)
    r = np.arange(n)
    cols = np.concatenate((state.pq_to_columns(p, q), state.pq_to_columns(r[None], ((r + 1) % n)[None])))
    g = np.random.default_rng(n + moves)
    mv = np.stack((g.integers(-1, 5, moves), g.integers(-1, 2 * n + 1, moves), g.integers(0, 2 * n, moves)), 1)
    mv = mv.astype(np.int32)
    dE, bad = gpu_delta.swap_deltas(cols, mv, badness=True)
    want, want_bad = gpu_delta.swap_deltas(cols, mv, badness=True, pairs=True)
    assert np.array_equal(dE, want) and np.array_equal(bad, want_bad)
    assert np.array_equal(gpu_delta.swap_deltas(cols, mv), want)
