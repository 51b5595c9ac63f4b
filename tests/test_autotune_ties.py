"""Pairs of (threads per chain, chains per CTA) that are the same launch differ by noise only: the tuner keeps the
narrowest width, whose chains per CTA are bounded least, whichever of them the noise favours."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import autotune


class Chains:
    def __init__(self, L, ladders):
        self.L = L
        self.ladder_n_host = np.full(ladders, 75, np.int32)
        self.cols = np.zeros((L * ladders, 150), np.int16)

    def default_chains_per_block(self, threads_per_chain=32):
        return 16 // (threads_per_chain // 32)


@pytest.mark.parametrize("favoured", [32, 64, 128, 256])
@pytest.mark.parametrize("best_cpb", [2, 4])
def test_noise_does_not_choose_the_width(favoured, best_cpb, monkeypatch):
    monkeypatch.setattr(autotune, "_clone", lambda ch, rows=None: ch)

    def seconds(ch, sweeps, *, exchange_every, cpb, ladder_sweeps=None, tpc=32):
        return (1.0 + 0.1 * (cpb != best_cpb)) * (1.0 - 0.0002 * (tpc == favoured))

    monkeypatch.setattr(autotune, "_timed", seconds)
    tune = autotune.autotune(Chains(16, 8), probe_sweeps=4, exchange_every=2)
    assert (tune.threads_per_chain, tune.chains_per_block) == (32, best_cpb)
    assert set(tune.candidates) == {f"{t}x{c}" for t, c in autotune._shapes(16, 8)}


def test_a_wider_shape_that_is_faster_is_kept(monkeypatch):
    monkeypatch.setattr(autotune, "_clone", lambda ch, rows=None: ch)
    monkeypatch.setattr(autotune, "_timed", lambda ch, sweeps, *, exchange_every, cpb, ladder_sweeps=None, tpc=32:
                        1.0 - 0.02 * (tpc == 128))
    assert autotune.autotune(Chains(16, 8), probe_sweeps=4, exchange_every=2).threads_per_chain == 128
