"""States with columns at or beyond n (below the largest grid's 75), and mutation of any columns at all: nothing
in these calls needs the columns to lie in the state's own grid, and they count them as they are."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import _lib, accelerated, gpu, gpu_delta, state, tempering

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


@pytest.mark.parametrize("bad_bias", [0, 85])
def test_tempering(bad_bias, oracle, cuda):
    """Chains whose columns were set by hand: the walk of the oracle, and no error bit."""
    import torch

    n, L = 20, 8
    p, q = state.seeded_population(n, L)
    ch = tempering.TemperingChains(state.pq_to_columns(p, q), np.geomspace(0.1, 4.0, L), 7, ladder_size=L)
    cols = state.pq_to_columns(3 * p, 3 * q)
    E, bad = gpu.score_columns_gpu(cols, badness=True)
    ch.cols[:, :2 * n] = torch.from_numpy(cols).cuda()
    ch.badness_dev[:, :2 * n] = torch.from_numpy(bad).cuda()
    ch.energy.copy_(torch.from_numpy(E))
    ch.best_energy.copy_(ch.energy)
    ch.best_cols.copy_(ch.cols)
    g = lambda x: x.cpu().numpy()  # noqa: E731
    take = lambda: {"cols": g(ch.cols).astype(np.int32), "bad": g(ch.badness_dev), "E": g(ch.energy),  # noqa: E731
                    "bestE": g(ch.best_energy), "best_cols": g(ch.best_cols).astype(np.int32),
                    "temp_of": g(ch.temp_of), "chain_at": g(ch.chain_at), "counter": g(ch.counter).astype(np.uint64),
                    "accepted": g(ch.accepted_dev).astype(np.uint32), "ladder_n": g(ch.ladder_n),
                    "ladder_round": g(ch.ladder_round).astype(np.uint32),
                    "ladder_exch": g(ch.ladder_exchanges).astype(np.uint32)}
    before = take()
    ch.run(30, exchange_every=15, graph=False, bad_bias=bad_bias)
    want = oracle.temper_run(before, ladder_size=L, acc=g(ch.acc_table).view(np.uint32),
                             exch=g(ch.exch_table).view(np.uint32), seed=ch.seed, rounds=2, round_sweeps=15,
                             bad_bias=bad_bias)
    after = take()
    for k in after:
        assert np.array_equal(after[k].astype(np.int64), np.asarray(want[k]).astype(np.int64)), k
    assert after["accepted"].sum() > 0 and int(ch.error_word.item()) == 0


@pytest.mark.parametrize("parents", [3, 200])  # badness sums staged in shared memory, and not
@pytest.mark.parametrize("shift", [0, 40000, -70000, 1 << 30])
def test_mutation_returns_any_columns(parents, shift, oracle, cuda):
    """Draws and swaps depend on which columns are equal, not on their values."""
    import torch

    n, population = 75, 700
    p, q = state.seeded_population(n, parents)
    bad = gpu.score_population_gpu(p, q, badness=True)[1]
    args = dict(quality_count=max(1, parents // 4), population=population, active_strength=4, max_strength=9,
                bad_bias=85, seed=11, generation=3)
    want_p, want_q = oracle.beam_mutate(p + shift, q + shift, bad, **args)
    dp, dq, db = (torch.from_numpy(np.ascontiguousarray(x, dtype=np.int32)).cuda() for x in (p + shift, q + shift, bad))
    cp = torch.empty((population, n), dtype=torch.int32, device="cuda")
    cq = torch.empty_like(cp)
    _lib.call("n3_beam_mutate", _lib.ptr(dp), _lib.ptr(dq), _lib.ptr(db), parents, args["quality_count"], n, population,
              args["active_strength"], args["max_strength"], args["bad_bias"], args["seed"], args["generation"],
              _lib.ptr(cp), _lib.ptr(cq), _lib.stream_ptr())
    assert np.array_equal(cp.cpu().numpy(), want_p) and np.array_equal(cq.cpu().numpy(), want_q)
