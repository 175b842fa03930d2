"""Crowded levels of long tapes: a frame that one block per cell could evaluate
succeeds whatever the sizes of the operand log's arena and of the work lists,
wherever its items are sent, and equals the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import assert_cells_equal
from temporalsetinversion_b200 import Device, Scene, Tape, api, scenes

TIMES = [0.0, 0.03, 0.05]


def run(dev, tape, p, threshold=None, parents=1, times=TIMES):
    t = Tape.upload(dev, tape)
    t.narrow_parents = parents
    if threshold is not None:
        t.wide_threshold = threshold
    gs, os_ = Scene(dev, t, p), oracle.Scene(tape, p)
    stats = None
    for time in times:
        stats = gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())
    return stats


def steep(n: int) -> np.ndarray:
    """A union of moving spheres scaled down and up again by more than the
    range of f32: every sensitivity is infinite at the last product of the
    reverse pass, so pruned tapes are run again in full."""
    body, last = scenes.csg(n, 3, 0.9).rsplit("  ret float %", 1)
    k = int(last.split()[0])
    chain = scenes.IRBuilder()
    chain.next = k + 1
    v = "%%%d" % k
    for i in range(14):
        v = chain.mul(v, 2.5e-6 if i < 7 else 4.0e5)
    text = body + "\n".join(chain.lines) + "\n  ret float %s\n}\n" % v
    return api.IR.new(text).gpu_instructions


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["swept", "normals"])
def test_unpruned_long_tapes_need_no_log(kind):
    """Derivatives in every cell of a 1177-instruction tape, no pruning, and
    an arena of 64 KB: less than one cell's log."""
    tape = api.IR.new(scenes.csg(64, 3, 0.9)).gpu_instructions
    p = dict(localsubdiv=9, pruning=0, delta=0.02)
    p.update(dict(swept_volume=1, swept_dt=0.05) if kind == "swept" else dict(normal_viz=1, fast_normals=0))
    with Device(log_arena_bytes=1 << 16) as dev:
        run(dev, tape, api.default_params(**p), times=TIMES[:2])


@pytest.mark.gpu
@pytest.mark.parametrize("parents", [1, 4])
@pytest.mark.parametrize("n,localsubdiv", [(64, 9), (330, 7), (600, 7)])
def test_second_runs_on_the_full_tape_need_no_log(n, localsubdiv, parents):
    """Cells of crowded levels with infinite sensitivities, on full tapes of
    1191, 6 and 11 thousand instructions, and the same arena.  (The threshold
    is below every pruned tape's length: no item is a short one.)"""
    tape = steep(n)
    with Device(log_arena_bytes=1 << 16) as dev:
        st = run(dev, tape, api.default_params(localsubdiv=localsubdiv, delta=0.02, normal_viz=1, fast_normals=0), 20, parents)
        assert st.prune_fallbacks > 0


@pytest.mark.gpu
def test_long_items_find_room_in_either_list():
    """Work lists a tenth too small for the busiest level's items in one list
    alone, all of them long: the other list takes the rest."""
    tape = api.IR.new(scenes.csg(48, 3, 0.9)).gpu_instructions
    assert len(tape) < 1000
    p = api.default_params(localsubdiv=9, pruning=0, delta=0.02)
    with Device() as dev:
        s = Scene(dev, Tape.upload(dev, tape), p)
        most = max(s.invert(time).items_high_water for time in TIMES[:2])
    assert most > 100
    with Device(work_item_capacity=int(0.9 * most)) as dev:
        run(dev, tape, p, times=TIMES[:2])
