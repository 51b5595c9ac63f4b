"""Moves by pairs of histograms and by the cover table where they can go wrong: every number of slots a
lane may hold, long lines (4-bit counters wrap, the move is counted again; cover entries in the
thousands), cold and hot chains of one ladder, launches too short for a cover table."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu, gpu_device_search, learned, state, tempering

pytestmark = pytest.mark.gpu


def snapshot(ch) -> dict:
    g = lambda x: x.cpu().numpy()  # noqa: E731
    return {"cols": g(ch.cols).astype(np.int32), "bad": g(ch.badness_dev), "E": g(ch.energy),
            "bestE": g(ch.best_energy), "best_cols": g(ch.best_cols).astype(np.int32), "temp_of": g(ch.temp_of),
            "chain_at": g(ch.chain_at), "counter": g(ch.counter).astype(np.uint64),
            "accepted": g(ch.accepted_dev).astype(np.uint32), "ladder_n": g(ch.ladder_n),
            "ladder_round": g(ch.ladder_round).astype(np.uint32),
            "ladder_exch": g(ch.ladder_exchanges).astype(np.uint32)}


def diagonals(n: int, count: int):
    """Two neighbouring diagonals (wrapped), shifted from state to state: lines of n - 1 and n points."""
    r = np.arange(n)
    p = np.stack([(r + s) % n for s in range(count)]).astype(np.int32)
    q = np.stack([(r + s + 1) % n for s in range(count)]).astype(np.int32)
    return state.pq_to_columns(p, q)


def run_and_replay(columns, temps, L, rounds, sweeps, bad_bias):
    from oracle import oracle

    ch = tempering.TemperingChains(columns, np.tile(temps, len(columns) // L), 77, ladder_size=L)
    before = snapshot(ch)
    ch.run(rounds * sweeps, exchange_every=sweeps, graph=False, bad_bias=bad_bias)
    ref = oracle.temper_run(before, ladder_size=L, acc=ch.acc_table.cpu().numpy().view(np.uint32),
                            exch=ch.exch_table.cpu().numpy().view(np.uint32), seed=ch.seed, rounds=rounds,
                            round_sweeps=sweeps, bad_bias=bad_bias)
    after = snapshot(ch)
    for k in after:
        assert np.array_equal(np.asarray(after[k]).astype(np.int64), np.asarray(ref[k]).astype(np.int64)), k
    assert int(ch.error_word.item()) == 0
    ch.validate()
    return after


@pytest.mark.parametrize("bad_bias", [0, 85])
@pytest.mark.parametrize("n", [3, 5, 16, 17, 32, 33, 48, 49, 64, 65, 74])
def test_every_number_of_slots_a_lane_holds(n, bad_bias, oracle, cuda):
    """Temperatures from below to above the cover table's, three rounds of at least 400 proposals."""
    p, q = state.seeded_population(n, 8)
    sweeps = max(1, -(-400 // (2 * n)))
    after = run_and_replay(state.pq_to_columns(p, q), np.geomspace(0.1, 6.0, 8), 8, 3, sweeps, bad_bias)
    assert after["accepted"].sum() > 0


@pytest.mark.parametrize("n,rounds", [(40, 2), (75, 2), (75, 1)])
def test_long_lines(n, rounds, oracle, cuda):
    """Diagonal states: sums far above what 4-bit counters hold, and cover entries of C(n - 1, 2)."""
    after = run_and_replay(diagonals(n, 8), np.geomspace(0.3, 400.0, 8), 8, rounds, 4, 0)
    assert after["accepted"].min() > 0


@pytest.mark.parametrize("n", [20, 75])
def test_beam_children_of_dense_parents(n, cuda):
    base = diagonals(n, 2).reshape(2, n, 2).astype(np.int32)
    beam = gpu_device_search.DeviceBeam(n, seed=3, population=300, elite_size=16, max_strength=6, energy_window=9,
                                        bad_bias=85, history_len=4)
    beam.init(base)
    for g in (1, 2):
        beam.generation(g)
        beam.read_status()  # raises if a maintained badness failed its check
        s, b = gpu.score_population_gpu(beam.child_p, beam.child_q, badness=True)
        assert bool((s == beam.child_scores).all()) and bool((b == beam.child_badness).all())


def test_learned_moves_on_dense_states(cuda):
    ch = tempering.TemperingChains(diagonals(75, 16), np.geomspace(0.3, 300.0, 16), 5, ladder_size=16)
    lp = learned.LearnedProposal(ch, seed=2, ring_capacity=4096, moves=16)
    for _ in range(6):
        lp.step()
    assert int(ch.accepted_dev.sum().item()) > 0 and int(ch.error_word.item()) == 0
    ch.validate()
