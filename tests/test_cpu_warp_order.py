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


def block_heads(text: str, at: int) -> list:
    """What stands before each open brace around a place, from the inside."""
    heads, depth = [], 0
    for i in range(at - 1, -1, -1):
        if text[i] == "}":
            depth += 1
        elif text[i] == "{":
            if depth == 0:
                heads.append(re.split(r"[;{}]", text[:i])[-1])
            else:
                depth -= 1
    return heads


def test_a_list_that_grows_is_read_once_a_warp():
    """goes_wide reads the length of a list that other blocks add to: two lanes
    may read different lengths, so it is asked by one thread alone, or the
    warp goes on with one lane's answer (else its lanes part before barriers
    and shuffles of the whole warp)."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "refine.cu").read_text())
    places = [m.start() for m in re.finditer(r"(?<!bool )\bgoes_wide\(", text)]
    assert len(places) >= 3
    for at in places:
        heads = block_heads(text, at)
        alone = any(re.search(r"if \((k|tid|lane) == 0\b", h) for h in heads)
        assert alone or text[:at].endswith("__shfl_sync(FULL_MASK, "), text[at - 200:at + 60]
