"""The checked score in one kernel (many states) against the same states in small batches, which take
the two kernels: sizes about the rule's, ragged shares, invalid states among valid ones."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,states", [(44, 1184), (55, 1300), (56, 2047), (75, 1200), (75, 9001)])
@pytest.mark.parametrize("badness", [True, False])
def test_one_kernel_agrees_with_two(n, states, badness, cuda):
    p, q = state.seeded_population(n, 300)
    cols = np.resize(state.pq_to_columns(p, q), (states, 2 * n))
    cols[7, 11] = n           # off the state's grid
    cols[450, 3] = -2
    cols[451, 0] = 120        # off every grid
    cols[states - 1, 5] = cols[states - 1, 4]
    cols[600] = np.repeat(np.arange(n), 2) // 2 + np.tile((0, n // 2), n)  # long lines
    got = gpu.score_checked_gpu(cols, raise_on_mismatch=False, badness=badness)
    parts = [gpu.score_checked_gpu(cols[i:i + 500], raise_on_mismatch=False, badness=badness)
             for i in range(0, states, 500)]
    assert np.array_equal(got.scores, np.concatenate([x.scores for x in parts]))
    if badness:
        assert np.array_equal(got.badness, np.concatenate([x.badness for x in parts]))
    assert got.mismatches == sum(x.mismatches for x in parts)
    assert got.error_word == np.bitwise_or.reduce([x.error_word for x in parts])
