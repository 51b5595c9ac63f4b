"""The error bits of the slope and checked scores: a row whose columns both lie off the grid on one side counts
as a duplicate point too, in every batch size."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 44, 75])
@pytest.mark.parametrize("states", [1, 300, 1300])
@pytest.mark.parametrize("pair,bits", [((-1, 0), 3), ((-4, -7), 3), ((0, 1), 0), ((2, 2), 2), ((3, -1), 1)])
def test_bits(n, states, pair, bits, cuda):
    p, q = state.seeded_population(n, 1)
    cols = np.resize(state.pq_to_columns(p, q), (states, 2 * n))
    cols[states // 2, 6:8] = pair
    beyond = cols.copy()
    beyond[states // 2, 6:8] = [n - 1 - c for c in pair]  # the same beyond the other edge
    for c in (cols, beyond):
        got = gpu.score_checked_gpu(c, raise_on_mismatch=False)
        assert got.error_word == bits and got.mismatches == (bits != 0)
        assert (got.scores[states // 2] == -1) == (bits != 0)
