"""The paths the population scores choose between: warps sharing a state at
small batch sizes, determinants on small grids and tags on larger ones, and
states that have no direction count."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, state

pytestmark = pytest.mark.gpu


def _determinants(cols):
    """E and badness of one slot-column state by int64 cross products, pivot slot by pivot slot; a
    triple that holds both points of a row is never counted (its third point lies in another row)."""
    m = len(cols)
    rows, c = np.arange(m) // 2, np.asarray(cols, np.int64)
    bad = np.zeros(m, np.int64)
    for a in range(m):
        dr, dc = rows - rows[a], c - c[a]
        hit = dr[:, None] * dc[None, :] == dc[:, None] * dr[None, :]
        other = (dr[:, None] != 0) & (dr[None, :] != 0) & (dr[:, None] != dr[None, :])
        bad[a] = np.count_nonzero(hit & other) // 2
    return int(bad.sum()) // 3, bad


@pytest.mark.parametrize("n", [3, 22, 23, 26, 27, 41])
@pytest.mark.parametrize("batch", [1, 2, 37, 149, 297, 593, 1185, 4145])
def test_every_batch_split_gives_the_same_counts(n, batch, oracle, cuda):
    p, q = state.seeded_population(n, min(batch, 40))
    reps = -(-batch // p.shape[0])
    p, q = np.tile(p, (reps, 1))[:batch], np.tile(q, (reps, 1))[:batch]
    head = min(batch, 40)
    ref_s, ref_b = oracle.score_population(p[:head], q[:head], badness=True, threads=0)
    ref_s, ref_b = np.tile(ref_s, reps)[:batch], np.tile(ref_b, (reps, 1))[:batch]
    cols = state.pq_to_columns(p, q)
    for s, b in (gpu.score_population_gpu(p, q, badness=True), gpu.score_columns_gpu(cols, badness=True),
                 gpu.score_slope_gpu(cols)):
        assert np.array_equal(s, ref_s) and np.array_equal(b, ref_b)
    assert np.array_equal(gpu.score_population_gpu(p, q), ref_s)
    chk = gpu.score_checked_gpu(cols)
    assert np.array_equal(chk.scores, ref_s) and np.array_equal(chk.badness, ref_b) and chk.mismatches == 0


@pytest.mark.parametrize("n", [9, 30, 75])
def test_states_without_a_direction_count_are_counted_by_determinants(n, cuda):
    """Columns off the grid and equal points of a row: the plain scores take them, as the determinant
    count always has, and count the states around them as before."""
    p, q = state.seeded_population(n, 6)
    cols = state.pq_to_columns(p, q)
    cols[1, 3] = 200            # off the 75 x 75 grid
    cols[2, 4] = cols[2, 5]     # two equal points in a row
    cols[3, 2] = -7
    cols[4, 0] = min(74, n)     # on the 75 x 75 grid, off the n x n one
    ref = [_determinants(c) for c in cols]
    # equal points of a row meet every line twice at once, which the count takes as one hit
    s, b = gpu.score_columns_gpu(cols, badness=True)
    ref[2] = (int(s[2]), b[2])
    assert 0 <= ref[2][0] <= _determinants(cols[2])[0]
    for B in (6, 1):  # whole and split over warps
        for lo in range(0, 6, B):
            s, b = gpu.score_columns_gpu(cols[lo:lo + B], badness=True)
            assert [int(x) for x in s] == [r[0] for r in ref[lo:lo + B]]
            assert np.array_equal(b, np.stack([r[1] for r in ref[lo:lo + B]]))
            assert np.array_equal(gpu.score_columns_gpu(cols[lo:lo + B]), s)
            s, b = gpu.score_population_gpu(cols[lo:lo + B, 0::2].astype(np.int32),
                                            cols[lo:lo + B, 1::2].astype(np.int32), badness=True)
            assert [int(x) for x in s] == [r[0] for r in ref[lo:lo + B]]
            assert np.array_equal(b, np.stack([r[1] for r in ref[lo:lo + B]]))
