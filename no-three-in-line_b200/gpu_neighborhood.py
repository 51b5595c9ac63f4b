"""Four-cycle and double-switch neighbourhood scans (drop-in for
``no_three_75.gpu_neighborhood``).

``best_four_cycle`` / ``best_double_switch`` keep the reference's signatures
and results (src/no_three_75/gpu_neighborhood.py:70-211): every candidate
through the anchor slot in the reference's enumeration order, the first
lowest-scoring legal one kept if it improves on the state, the same
``evaluated`` / ``legal`` counts.  The reference builds every candidate state
on the host (3.1 M states at n = 75 for a four-cycle scan) and rescores each in
full on the GPU; here one kernel scores every candidate exactly from a cover
table and direction histograms around the positions that three of its slots fix
(libn3 ``n3_neighborhood_scan``), and the host only decodes the winner and
checks it with the two independent device counts.  ``batch_size`` is accepted
for the reference's signature; the scan needs no batching.
"""
from __future__ import annotations

import ctypes
import time
from dataclasses import dataclass
from itertools import permutations
from math import comb

import numpy as np

from . import _lib
from .accelerated import score_and_badness
from .state import PairPermutations, points_to_permutations

_BASE = 1 << 30  # above any score, so that no candidate's goes below 0

_lib.register("n3_neighborhood_scan", [_lib._P, _lib._P, _lib._I, _lib._I, _lib._I64, _lib._P, _lib._P, _lib._P])


@dataclass(frozen=True)
class FourCycleResult:
    """gpu_neighborhood.py:14-21."""
    state: PairPermutations
    score: int
    anchor_index: int
    evaluated: int
    legal: int
    elapsed_seconds: float


@dataclass(frozen=True)
class DoubleSwitchResult:
    """gpu_neighborhood.py:24-31."""
    state: PairPermutations
    score: int
    anchor_index: int
    evaluated: int
    legal: int
    elapsed_seconds: float


def _values_state(values: np.ndarray) -> PairPermutations:
    """gpu_neighborhood.py:34-37."""
    n = values.shape[0]
    points = [(row, column) for row, pair in enumerate(values.tolist()) for column in pair]
    return points_to_permutations(points, n)


def bad_anchor_indices(state: PairPermutations, limit: int) -> list[int]:
    """gpu_neighborhood.py:128-132: slots by decreasing badness, then index."""
    _, badness = score_and_badness(np.asarray(state.P, dtype=np.int32), np.asarray(state.Q, dtype=np.int32))
    return sorted(range(2 * state.n), key=lambda index: (-int(badness[index]), index))[:limit]


def _scan(state: PairPermutations, anchor_index: int):
    state.validate()
    n = state.n
    if not (0 <= anchor_index < 2 * n):
        raise ValueError("anchor index outside point slots")
    if not 5 <= n <= _lib.MAX_N:
        raise ValueError(f"n={n} outside [5, {_lib.MAX_N}]")
    t = _lib.torch()
    device = _lib.require_device()
    pq = np.asarray((state.P, state.Q), dtype=np.int32)
    on_device = t.from_numpy(pq).to(device)
    dp = _lib.ptr(on_device)
    dq, stream = dp + 4 * n, _lib.stream_ptr()
    # The scan runs with _BASE in place of the state's score, so that the score
    # follows it on the stream and both come back in one copy.
    out = t.empty(5, dtype=t.int64, device=device)
    dst = _lib.ptr(out)
    _lib.call("n3_neighborhood_scan", dp, dq, n, int(anchor_index), _BASE, dst, dst + 16, stream)
    _lib.call("n3_score_population", dp, dq, 1, n, dst + 32, None, stream)
    best4, best2, legal4, legal2, score = (int(x) for x in out.cpu().numpy().view(np.uint64))
    base_score = score & 0xFFFFFFFF
    rebase = (base_score - _BASE) << 32
    return n, pq[0], pq[1], base_score, (best4 + rebase, legal4), (best2 + rebase, legal2)


def _slot_set(n: int, anchor: int, combo_layers: int):
    """Decode (row triple, layer choice) number k of gpu_neighborhood.py:108-110."""
    rank, layers = divmod(combo_layers, 8)
    rows, low = [], 0
    for left in (2, 1, 0):  # rows still to choose after this one
        while (later := comb(n - 2 - low, left)) <= rank:
            rank -= later
            low += 1
        rows.append(low if low < anchor // 2 else low + 1)
        low += 1
    return tuple(2 * r + ((layers >> (2 - i)) & 1) for i, r in enumerate(rows))


def _apply(base: np.ndarray, targets, sources) -> np.ndarray:
    flat = base.reshape(-1)
    changed = flat.copy()
    changed[list(targets)] = flat[list(sources)]
    return changed.reshape(base.shape)


def _verified(values: np.ndarray, score: int, what: str) -> None:
    """The reference re-scores the winner on the CPU (gpu_neighborhood.py:101-103);
    here both independent device counts (determinant and slope) must give it."""
    from .gpu import score_checked_gpu
    from .state import pq_to_columns

    checked = score_checked_gpu(pq_to_columns(values[None, :, 0], values[None, :, 1]), raise_on_mismatch=False,
                                badness=False)
    exact = int(checked.scores[0])
    if exact != score or checked.mismatches:
        raise AssertionError(f"GPU {what} score {score} != full score {exact}")


def best_four_cycle(state: PairPermutations, anchor_index: int, *, batch_size: int = 32768) -> FourCycleResult:
    """gpu_neighborhood.py:70-125."""
    started = time.perf_counter()
    n, p, q, base_score, (key, legal), _ = _scan(state, anchor_index)
    base = np.column_stack((p, q)).astype(np.int32)
    combos = (n - 1) * (n - 2) * (n - 3) // 6
    evaluated = combos * 8 * 6
    best_score, best_values = base_score, base
    if legal and (key >> 32) < base_score:
        idx = key & 0xFFFFFFFF
        order = list(permutations(_slot_set(n, anchor_index, idx // 6)))[idx % 6]
        targets = (anchor_index,) + tuple(order)
        best_score = int(key >> 32)
        best_values = _apply(base, targets, targets[1:] + targets[:1])
        _verified(best_values, best_score, "four-cycle")
    return FourCycleResult(_values_state(best_values), best_score, anchor_index, evaluated, legal,
                           time.perf_counter() - started)


def best_double_switch(state: PairPermutations, anchor_index: int, *, batch_size: int = 32768) -> DoubleSwitchResult:
    """gpu_neighborhood.py:135-211."""
    started = time.perf_counter()
    n, p, q, base_score, _, (key, legal) = _scan(state, anchor_index)
    base = np.column_stack((p, q)).astype(np.int32)
    combos = (n - 1) * (n - 2) * (n - 3) // 6
    evaluated = combos * 8 * 3
    best_score, best_values = base_score, base
    if legal and (key >> 32) < base_score:
        idx = key & 0xFFFFFFFF
        a, b, c = _slot_set(n, anchor_index, idx // 3)
        sources = ((a, anchor_index, c, b), (b, c, anchor_index, a), (c, b, a, anchor_index))[idx % 3]
        best_score = int(key >> 32)
        best_values = _apply(base, (anchor_index, a, b, c), sources)
        _verified(best_values, best_score, "double-switch")
    return DoubleSwitchResult(_values_state(best_values), best_score, anchor_index, evaluated, legal,
                              time.perf_counter() - started)
