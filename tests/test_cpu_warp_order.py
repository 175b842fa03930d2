"""The decoded instructions that the lanes of a warp hand to one another through
shared memory: wherever a lane stores its own, a warp barrier stands before
the first that is read back (votes and shuffles order no memory), and another
between the last that is read and the next store.  Read from the sources: a
missing barrier shows in no result until a compiler or a GPU reorders the
accesses."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "temporalsetinversion_b200" / "csrc"
CALLS = re.compile(r"\b(prog_st|prog_ld|__syncwarp)\(")


def calls(name: str) -> list:
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    text = re.sub(r"__forceinline__ \w+ prog_(st|ld)\(", "(", text)  # the definitions
    return [m.group(1) for m in CALLS.finditer(text)]


@pytest.mark.parametrize("name", ["narrow_interp.cuh", "point_tape.cuh", "refine.cu"])
def test_a_barrier_stands_between_stores_and_loads(name):
    seq = calls(name)
    stores = [i for i, c in enumerate(seq) if c == "prog_st"]
    assert stores
    for i in stores:
        assert seq[i + 1] == "__syncwarp" and seq[i - 1] == "__syncwarp", (name, seq[max(0, i - 2):i + 3])
        assert "prog_ld" in seq[i + 2:]
