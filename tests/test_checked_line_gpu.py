"""The checked score about the line between its one kernel and its two, on the grids where that line has two ends:
the same scores, badness and verdicts as the counts alone."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [43, 44, 48, 49])
@pytest.mark.parametrize("per_sm,more", [(8, -1), (8, 0), (8, 1), (20, 0), (20, 1)])
def test_both_sides(n, per_sm, more, cuda):
    import torch

    states = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    p, q = state.seeded_population(n, 200)
    few = state.pq_to_columns(p, q)
    few[77, 3] = few[77, 2]
    few[111, 9] = n
    cols = np.resize(few, (states, 2 * n))
    E, _ = gpu.score_determinants_gpu(few, badness=True)
    slope, bad = gpu.score_slope_gpu(few)
    E[[77, 111]] = -1
    assert np.array_equal(E, slope)
    for badness in (True, False):
        got = gpu.score_checked_gpu(cols, raise_on_mismatch=False, badness=badness)
        want = np.resize(E, states)
        assert np.array_equal(got.scores, want) and got.mismatches == int((want < 0).sum()) and got.error_word == 3
        if badness:
            assert np.array_equal(got.badness, np.resize(bad, (states, 2 * n)))
