"""Kernels that begin with chain_begin() may be on the SMs while the kernels before them still write, so no
load of theirs may take the read-only path, whose data must not change while the kernel lives: no __ldg and
no `const T* __restrict__` for global memory in them or in the functions that they hand it to."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "no-three-in-line_b200" / "csrc"
# Shared memory, or tables that are built once per device before any kernel reads them.
CONSTANT = {"lut", "lut4", "prim4", "recip", "dir4_", "cs", "bs", "hist", "T", "occ", "bits", "scratch", "rows4"}


def functions(text: str) -> list[tuple[str, str, str]]:
    """(name, parameters, body) of every function definition."""
    out = []
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"\b(\w+)\(([^;{}]*?)\)\s*\{", text):
        depth, at = 1, m.end()
        while depth and at < len(text):
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        if m.group(1) not in ("if", "for", "while", "switch"):
            out.append((m.group(1), m.group(2), text[m.end():at]))
    return out


def chained(funcs) -> set[str]:
    """Names of the kernels that wait in chain_begin(), themselves or through a function, and of all they call."""
    calls = {name: set(re.findall(r"\b(\w+)\s*(?:<[^<>;]*>)?\(", body)) for name, _, body in funcs}
    waits = {name for name, _, body in funcs if "chain_begin()" in body}
    while more := {n for n, c in calls.items() if c & waits} - waits:
        waits |= more
    while more := {c for n in waits for c in calls.get(n, ()) if c in calls} - waits:
        waits |= more
    return waits


@pytest.mark.parametrize("name", ["mlp.cu", "beam.cu"])
def test_no_read_only_loads_in_chained_kernels(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    funcs = functions(text)
    names = chained(funcs)
    assert len(names) >= 5
    for function, parameters, body in funcs:
        if function not in names:
            continue
        assert "__ldg" not in body, function
        for pointer in re.findall(r"\bconst\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", parameters):
            assert pointer in CONSTANT, (function, pointer)


def test_chained_launches_only_of_kernels_that_wait():
    """launch_chained lets a kernel start early, so each kernel given to it must wait."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        funcs = functions(text)
        names = chained(funcs)
        for kernel in re.findall(r"launch_chained\(\s*\"[^\"]*\",\s*(?:\w+::)*(\w+)", text):
            assert kernel in names, (path.name, kernel)
