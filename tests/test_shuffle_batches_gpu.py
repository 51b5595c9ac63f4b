"""The shuffle's draws where a batch of MT19937 blocks sized for them runs out before the last step, for
every size of batch from one block up: rare draws (found by replaying the batches on the host), each
followed by more shuffles, which continue from the state it leaves."""
from __future__ import annotations

from random import Random

import numpy as np
import pytest

from no_three_in_line_b200 import gpu_device_search as gds

pytestmark = pytest.mark.gpu
WORDS, BATCH = 624, 8


def first_batch(seed: int, count: int) -> tuple[int, int]:
    """(blocks of a fresh state's first batch, blocks that its draws need)."""
    left = count - 1
    blocks = min(BATCH, (left + left // 2 + 64) // WORDS + 1)
    rng, words = Random(seed), 0
    for i in range(left, 0, -1):
        words += 1
        while rng.getrandbits(32) >> (32 - (i + 1).bit_length()) > i:
            words += 1
    return blocks, -(-words // WORDS)


@pytest.mark.parametrize("seed,count,blocks", [(74698, 373, 1), (123873, 373, 1), (2124, 790, 2), (10956, 1205, 3),
                                               (12257, 1621, 4), (829, 2451, 6), (1208, 2869, 7)])
def test_a_batch_that_runs_out(seed, count, blocks, cuda):
    assert first_batch(seed, count) == (blocks, blocks + 1)
    counts = [count, 300, 5000, 17]
    for _ in range(3):  # the race this guards against depended on the order of warps
        rng = Random(seed)
        for c, got in zip(counts, gds.py_shuffle_steps_device(counts, seed)):
            want = [0] * c
            for i in range(c - 1, 0, -1):
                want[i] = rng._randbelow(i + 1)
            assert np.array_equal(got, want), c
