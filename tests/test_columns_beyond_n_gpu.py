"""States with columns at or beyond n (below the largest grid's 75): nothing in these calls needs the columns to
lie in the state's own grid, and they count them as they are."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import accelerated, gpu, gpu_delta, state

pytestmark = pytest.mark.gpu


def spread(n: int, count: int):
    """Two points a row in every third column of a grid of 3 n <= 75."""
    p, q = state.seeded_population(n, count)
    return 3 * p, 3 * q


@pytest.mark.parametrize("n", [8, 20, 25])
def test_partner_scores(n, oracle, cuda):
    import torch

    p, q = spread(n, 3)
    cols = state.pq_to_columns(p, q)
    E, bad = gpu.score_columns_gpu(cols, badness=True)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    runs = [(b, u) for b in range(3) for u in range(2 * n)] + [(b, 1) for b in (0, 2, 1)]  # long and short ones
    got = gpu_delta.two_switch_scores(dev(cols), dev(bad), dev(E), dev(np.asarray(runs, np.int32))).cpu().numpy()
    for (b, u), line in zip(runs, got):
        want = oracle.two_switches(p[b], q[b], u, int(E[b]), bad[b].astype(np.int64))
        legal = want < 1 << 59
        assert np.array_equal(line[legal], want[legal]) and (line[~legal] == gpu_delta.SENTINEL).all()
    one = accelerated.evaluate_two_switches(p[1], q[1], 3, int(E[1]), bad[1])
    assert np.array_equal(one, oracle.two_switches(p[1], q[1], 3, int(E[1]), bad[1].astype(np.int64)))
