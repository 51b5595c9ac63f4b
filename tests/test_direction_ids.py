"""The tag bytes that a warp of the slope count has room for, by the slots a lane holds, cover every direction that a
grid of that size has: ids are numbered by (dx, dy), dx >= 0, whatever dy."""
from __future__ import annotations

import re
from math import gcd
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "no-three-in-line_b200" / "csrc"


def directions(rows: int) -> int:
    """Primitive directions (dx, dy) with 0 <= dx < rows, |dy| < 75."""
    return 1 + sum(gcd(dx, abs(dy)) == 1 for dx in range(1, rows) for dy in range(-74, 75))


def test_tag_bytes_cover_the_directions():
    text = (CSRC / "score.cu").read_text()
    sizes = dict(re.findall(r"nt == (\d) \? (\d+)", text[text.index("int tag_ids(int nt)"):][:200]))
    assert set(sizes) == {"1", "2", "3"}
    for nt, size in sizes.items():
        assert directions(16 * int(nt)) <= int(size) < directions(16 * int(nt)) + 8
    total = int(re.search(r"kDirCount = (\d+)", (CSRC / "dirs.cuh").read_text()).group(1))
    assert directions(75) == total
