"""The determinant count on its own: every launch shape and both ways of counting against the oracle, and the
callers that name it use it, so that it never stands against itself."""
from __future__ import annotations

from random import Random

import numpy as np
import pytest

from no_three_in_line_b200 import _lib, gpu, precompute, state, tempering

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 22, 23, 27, 48, 75])
@pytest.mark.parametrize("states", [1, 297, 1185])  # a state per 16, 4 and 1 warps
def test_counts(n, states, oracle, cuda):
    p, q = state.seeded_population(n, 40)
    cols = np.resize(state.pq_to_columns(p, q), (states, 2 * n))
    E, bad = oracle.score_population(p, q, badness=True, threads=0)
    scores, badness = gpu.score_determinants_gpu(cols, badness=True)
    assert np.array_equal(scores, np.resize(E, states)) and np.array_equal(badness, np.resize(bad, (states, 2 * n)))
    assert np.array_equal(gpu.score_determinants_gpu(cols), scores)


def test_columns_off_every_grid(oracle, cuda):
    p, q = state.seeded_population(40, 3)
    p[1, 7], q[2, 0] = 3000, -5
    E, bad = oracle.score_population(p, q, badness=True, threads=0)
    scores, badness = gpu.score_determinants_gpu(state.pq_to_columns(p, q), badness=True)
    assert np.array_equal(scores, E) and np.array_equal(badness, bad)


def called(monkeypatch, run):
    names, call = [], _lib.call
    monkeypatch.setattr(_lib, "call", lambda name, *args: (names.append(name), call(name, *args))[1])
    run()
    return set(names)


def test_scorer_a_of_the_precomputation_benchmark(monkeypatch, cuda):
    s = state.random_state(30, Random(5))
    points = [(r, int(c)) for r in range(30) for c in (s.P[r], s.Q[r])]
    names = called(monkeypatch, lambda: precompute.benchmark_precomputation(30, points))
    assert {"n3_score_determinants", "n3_score_slope"} <= names
    assert not names & {"n3_score_population", "n3_score_columns"}


def test_reference_checkpoint(monkeypatch, tmp_path, cuda):
    """A checkpoint as the reference writes it is checked by determinants; a wrong badness is refused."""
    p, q = state.seeded_population(30, 8)
    cols = state.pq_to_columns(p, q)
    scores, bad = gpu.score_determinants_gpu(cols, badness=True)
    keep = dict(columns=cols.astype(np.int32), temperatures=np.geomspace(0.2, 4.0, 8), scores=scores, badness=bad,
                rngs=np.arange(8, dtype=np.uint64) + 5)
    np.savez(tmp_path / "a.npz", **keep)
    assert "n3_score_determinants" in called(monkeypatch, lambda: tempering.TemperingChains.restore(tmp_path / "a.npz"))
    bad = bad.copy()
    bad[3, 4] += 1
    np.savez(tmp_path / "b.npz", **dict(keep, badness=bad))
    with pytest.raises(AssertionError, match="determinant"):
        tempering.TemperingChains.restore(tmp_path / "b.npz")
