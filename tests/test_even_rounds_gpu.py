"""Batches just above what the warps of the GPU take at once, where the work is shared evenly instead of
leaving a few items to a round of their own."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, gpu_delta, state

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


@pytest.mark.parametrize("n", [3, 16, 17, 26, 32, 33, 48, 49, 75])
@pytest.mark.parametrize("states", [1, 149, 2368, 2369, 4144, 4145, 4300, 4736, 4737, 9000])
def test_slope_counts(n, states, cuda):
    """E, badness and error bits of every state, some of them without a line count."""
    p, q = state.seeded_population(n, 29)
    few = state.pq_to_columns(p, q)
    few[11, 1] = few[11, 0]
    few[23, 2 * n - 1] = -1
    cols = np.resize(few, (states, 2 * n))
    E, bad = gpu.score_determinants_gpu(few, badness=True)
    got, got_bad = gpu.score_columns_gpu(cols, badness=True)
    assert np.array_equal(got, np.resize(E, states)) and np.array_equal(got_bad, np.resize(bad, (states, 2 * n)))
    assert np.array_equal(gpu.score_columns_gpu(cols), got)
    E[[11, 23]], bad[[11, 23]] = -1, -1
    scores, badness = gpu.score_slope_gpu(cols)
    assert np.array_equal(scores, np.resize(E, states)) and np.array_equal(badness, np.resize(bad, (states, 2 * n)))
    wrong = int((np.resize(E, states) < 0).sum())
    for want_badness in (True, False):
        checked = gpu.score_checked_gpu(cols, raise_on_mismatch=False, badness=want_badness)
        assert np.array_equal(checked.scores, np.resize(E, states)) and checked.mismatches == wrong
        assert checked.error_word == (0 if states < 12 else 2 if states < 24 else 3)
        if want_badness:
            assert np.array_equal(checked.badness, np.resize(bad, (states, 2 * n)))
