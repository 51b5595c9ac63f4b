"""The beam selection's paths against the CPU oracle: windows larger than one table of the traced shuffle
holds, more keys than are sorted by counting, scores above the one-pass histogram's range and above 16
bits, populations that end inside a word."""
from __future__ import annotations

import numpy as np
import pytest

from no_three_in_line_b200 import gpu_device_search as gds
from no_three_in_line_b200 import state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,diagonal,population,elite,window,generations", [
    (7, False, 65536, 2048, 10**6, 2),   # the whole population in the window: the table in parts
    (16, False, 31000, 1100, 10**6, 2),
    (9, False, 33, 33, 3, 4),
    (23, False, 1025, 16, 0, 4),
    (40, True, 4097, 64, 50, 3),         # scores about 19,000
    (75, True, 2500, 70, 400, 3),        # about 130,000
])
def test_selection_matches_oracle(cuda, oracle, n, diagonal, population, elite, window, generations):
    if diagonal:
        p = np.arange(n, dtype=np.int32)
        q = (p + 1) % n
    else:
        p, q = (x[0] for x in state.seeded_population(n, 1))
    p, q = p.astype(np.int32), q.astype(np.int32)
    cfg = dict(seed=17, population=population, elite_size=elite, max_strength=5, energy_window=window)
    ref = oracle.beam_search(p, q, None, generations=generations, **cfg)
    beam = gds.DeviceBeam(n, bad_bias=85, history_len=generations, **cfg)
    beam.init(np.column_stack((p, q))[None])
    for g in range(1, ref["completed"] + 1):
        beam.generation(g)
        assert np.array_equal(beam.elite_scores.cpu().numpy(), ref["elite_scores"][g - 1]), g
        assert np.array_equal(beam.elite_p.cpu().numpy(), ref["elite_p"][g - 1]), g
        assert np.array_equal(beam.elite_q.cpu().numpy(), ref["elite_q"][g - 1]), g
