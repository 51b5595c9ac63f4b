"""The neighbourhood scan's paths: grids on both sides of the size rule, states with two points in every
column and others, row triples with shared columns; best candidate, its index and the legal counts
against every candidate state scored in full."""
from __future__ import annotations

from itertools import combinations, permutations, product

import numpy as np
import pytest

from no_three_in_line_b200 import _lib, gpu, gpu_neighborhood, state  # noqa: F401

pytestmark = pytest.mark.gpu


def brute(cols, anchor):
    """[(lowest score, first index), legal] of the four-cycles and of the double switches."""
    n = len(cols) // 2
    rows = [r for r in range(n) if r != anchor // 2]
    moves = ([], [])
    for triple in combinations(rows, 3):
        for layers in product((0, 1), repeat=3):
            a, b, c = (2 * r + l for r, l in zip(triple, layers))
            for order in permutations((a, b, c)):
                t = (anchor,) + order
                moves[0].append((t, t[1:] + t[:1]))
            for s in ((a, anchor, c, b), (b, c, anchor, a), (c, b, a, anchor)):
                moves[1].append(((anchor, a, b, c), s))
    out = []
    for kind in moves:
        t, s = (np.asarray([m[i] for m in kind]) for i in (0, 1))
        all_cols = np.repeat(cols[None], len(t), axis=0)
        np.put_along_axis(all_cols, t, cols[s], axis=1)
        legal = (cols[s] != cols[t ^ 1]).all(1)
        scores = gpu.score_columns_gpu(np.ascontiguousarray(all_cols[legal]))
        index = np.flatnonzero(legal)
        out.append(((int(scores.min()), int(index[scores.argmin()])) if len(index) else None, len(index)))
    return out


def scan(cols, anchor):
    import torch

    n = len(cols) // 2
    p, q = (torch.from_numpy(cols[k::2].astype(np.int32)).cuda() for k in (0, 1))
    base = int(gpu.score_columns_gpu(cols[None])[0])
    out = torch.empty(4, dtype=torch.int64, device="cuda")
    _lib.call("n3_neighborhood_scan", _lib.ptr(p), _lib.ptr(q), n, anchor, base, _lib.ptr(out), _lib.ptr(out) + 16,
              _lib.stream_ptr())
    v = [int(x) for x in out.cpu().numpy().view(np.uint64)]
    return [((v[i] >> 32, v[i] & 0xFFFFFFFF) if v[2 + i] else None, v[2 + i]) for i in (0, 1)]


@pytest.mark.parametrize("n", [5, 12, 13, 14, 18, 21])
def test_scan_matches_full_scores(n, cuda):
    p, q = state.seeded_population(n, 1)
    cols = state.pq_to_columns(p, q)[0]
    r = np.arange(n)
    diag = state.pq_to_columns(r[None].astype(np.int32), ((r + 1) % n)[None].astype(np.int32))[0]
    uneven = cols.copy()
    uneven[0::2], uneven[1::2] = r % 4, 4 + r % (n - 4)
    for c, anchors in ((cols, (0, n, 2 * n - 1)), (diag, (1, n)), (uneven, (2, 2 * n - 1))):
        for a in anchors:
            assert scan(c, a) == brute(c, a), a
