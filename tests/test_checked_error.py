"""The rule that decides a checked score, the same function on the host and in the kernels: a slip planted in
either count of E or in the badness raises the mismatch bit."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import _lib, state

MISMATCH = 4


def verdict(det: int, slope: int, badness=None) -> int:
    has = badness is not None
    return _lib.lib().n3_checked_error(int(det), int(slope), int(has), int(np.sum(badness)) if has else 0)


@pytest.mark.parametrize("n", [8, 20, 75])
def test_planted_slips_are_seen(n):
    from oracle import oracle

    p, q = state.seeded_population(n, 1)
    E, bad = oracle.score_and_badness(p[0], q[0])
    assert verdict(E, E) == 0 and verdict(E, E, bad) == 0
    assert verdict(E, E + 1) == MISMATCH and verdict(E + 1, E) == MISMATCH and verdict(E + 1, E, bad) == MISMATCH
    for slot in (0, n, 2 * n - 1):
        for by in (-1, 1, 3):
            slipped = np.asarray(bad).copy()
            slipped[slot] += by
            assert verdict(E, E, slipped) == MISMATCH
    assert verdict(0, 0, np.zeros(2 * n)) == 0 and verdict(0, 0, np.asarray([-1])) == MISMATCH
