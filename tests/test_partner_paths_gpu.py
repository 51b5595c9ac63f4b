"""The paths the partner scores choose between: runs of anchors of one state long enough for a cover
table, shorter ones, states whose columns do not hold two points each, equal columns, anchors out of
range; every score against the batched swap deltas, which share no code with them."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, gpu_delta, state

pytestmark = pytest.mark.gpu
SENT = gpu_delta.SENTINEL


def expected(cols, E, anchors, same_layer):
    """Scores by swap_deltas; equal columns give the state's own score, other illegal swaps the sentinel."""
    B, m = cols.shape
    rows, flat = [], []
    for b, u in anchors:
        vs = range(u & 1, m, 2) if same_layer else range(m)
        rows.append((b, u, list(vs) if 0 <= b < B and 0 <= u < m else []))
        flat += [(b, u, v) for v in rows[-1][2]]
    dE = iter(gpu_delta.swap_deltas(cols, np.asarray(flat, np.int32).reshape(-1, 3)).tolist() if flat else [])
    out = []
    for b, u, vs in rows:
        line = [SENT] * (m // 2 if same_layer else m)
        for w, v in enumerate(vs):
            d, c = next(dE), cols[b]
            if u // 2 != v // 2 and c[v] != c[u ^ 1] and c[u] != c[v ^ 1]:
                line[w] = int(E[b]) + (0 if c[u] == c[v] else d)
        out.append(line)
    return np.asarray(out)


def check(cols, anchors, cuda):
    import torch

    E, bad = gpu.score_columns_gpu(cols, badness=True)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    anchors = np.asarray(anchors, np.int32)
    for same_layer, call in ((False, gpu_delta.two_switch_scores), (True, gpu_delta.transposition_scores)):
        got = call(dev(cols), dev(bad), dev(E), dev(anchors)).cpu().numpy()
        assert np.array_equal(got, expected(cols, E, anchors.tolist(), same_layer)), same_layer


@pytest.mark.parametrize("n", [2, 3, 8, 17, 32, 33, 64, 75])
def test_runs_of_every_length(n, cuda):
    p, q = state.seeded_population(n, 5)
    cols = state.pq_to_columns(p, q)
    m = 2 * n
    anchors = [(0, u) for u in range(m)]                         # a whole state
    anchors += [(1, u % m) for u in range(7)] + [(2, u % m) for u in range(8)]  # about the line of the rule
    anchors += [(b, (3 * b + 1) % m) for b in (3, 4, 3, 4, 0)]   # single ones
    anchors += [(-1, 0), (9, 0), (4, -1), (4, m), (4, m - 1)]    # out of range
    check(cols, anchors, cuda)
    check(cols, anchors[:1], cuda)


def test_diagonals_and_uneven_columns(cuda):
    n = 40
    r = np.arange(n)
    diag = state.pq_to_columns(r[None].astype(np.int32), ((r + 1) % n)[None].astype(np.int32))
    uneven = diag.copy()
    uneven[0, 0::2] = r % 7          # many points in a few columns
    uneven[0, 1::2] = 7 + r % 11
    cols = np.concatenate((diag, uneven, diag))
    check(cols, [(b, u) for b in (0, 1, 2) for u in range(0, 2 * n, 3)] + [(1, 5), (0, 3)], cuda)


def test_a_cell_held_twice(cuda):
    """Two points in every column, but one cell twice: runs of a state's anchors and single ones agree."""
    import torch

    n = 40
    r = np.arange(n)
    cols = state.pq_to_columns(r[None].astype(np.int32), ((r + 1) % n)[None].astype(np.int32))
    cols[0, 11], cols[0, 9] = 5, 6   # rows 5 and 4 held columns 5, 6 and 4, 5
    cols = np.repeat(cols, 2, axis=0)
    E, bad = gpu.score_columns_gpu(cols, badness=True)
    runs = [(b, u) for b in (0, 1) for u in range(2 * n)]
    single = [(b, u) for u in range(2 * n) for b in (0, 1)]
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    for call in (gpu_delta.two_switch_scores, gpu_delta.transposition_scores):
        a, b = (call(dev(cols), dev(bad), dev(E), dev(np.asarray(x, np.int32))).cpu().numpy() for x in (runs, single))
        assert np.array_equal(a.reshape(2, 2 * n, -1), b.reshape(2 * n, 2, -1).transpose(1, 0, 2))
