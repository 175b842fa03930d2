"""The one-warp tape interpreter at the sizes where it can go wrong: tapes
whose length ends on, one before and one after a chunk of 32 instructions,
items of one, two and four parents (rows of 9, 17 and 32 columns), literals
beyond the clamp of `fix`, uploaded tapes whose use counts are wrong, and the
directed form against the block-wide interpreter."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import assert_cells_equal
from temporalsetinversion_b200 import Scene, Tape, api, scenes

TIMES = [0.0, 0.03, 0.05, 0.3]


def mixed_tape(length: int, seed: int) -> np.ndarray:
    """A union and intersection of moving spheres with every handler class in
    between, padded to `length` instructions (after the four arguments)."""
    rng = np.random.default_rng(seed)
    b = scenes.IRBuilder()

    def sphere():
        c = [float(x) for x in rng.uniform(-2.0, 2.0, 3)]
        m = b.mul(b.sin(b.add(b.T, float(rng.uniform(0, 6)))), 0.5)
        d = [b.sub(v, b.add(m, ck)) for v, ck in zip((b.X, b.Y, b.Z), c)]
        s = b.add(b.add(b.mul(d[0], d[0]), b.mul(d[1], d[1])), b.mul(d[2], d[2]))
        return b.sub(b.sqrt(s), float(rng.uniform(0.8, 1.8)))

    acc = sphere()
    k = 0
    while len(b.lines) + 20 < length:
        k += 1
        step = k % 7
        if step == 0:
            acc = b.sub(b.abs(b.add(acc, 0.4)), 0.4)
        elif step == 1:
            acc = b.min(acc, sphere())
        elif step == 2:
            acc = b.neg(b.neg(acc))
        elif step == 3:
            acc = b.mul(b.mul(acc, 2.5e-7), 4.0e6)   # a factor beyond the clamp, values far below it
        elif step == 4:
            acc = b.max(acc, b.neg(b.min(b.sub(1.0, b.mul(b.X, b.Y)), 2.5)))
        elif step == 5:
            acc = b.mul(acc, -1.5)
            acc = b.mul(acc, -0.5)
        else:
            acc = b.max(b.min(acc, 3.0), -3.0)
    while len(b.lines) + 1 < length:
        acc = b.add(acc, 0.0)
    tape = api.IR.new(b.text(acc)).gpu_instructions
    assert len(tape) == length + 4
    return tape


@pytest.mark.gpu
@pytest.mark.parametrize("parents", [1, 2, 4])
@pytest.mark.parametrize("length", [31, 32, 33, 63, 64, 65, 97, 160])
def test_chunk_edges_match_oracle(device, length, parents):
    tape = mixed_tape(length, length)
    p = api.default_params(localsubdiv=5, delta=0.02, pointsample=length % 2)
    t = Tape.upload(device, tape)
    t.narrow_parents = parents
    gs, os_ = Scene(device, t, p), oracle.Scene(tape, p)
    for time in TIMES:
        gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2])
def test_wrong_use_counts_match_oracle(device, seed):
    """Values with several users whose use count says one: the skip rule then
    resets sums, which no shortcut may leave out."""
    tape = mixed_tape(70, 100 + seed).copy()
    ou = tape["opcode_uses"]
    rng = np.random.default_rng(seed)
    pick = rng.uniform(size=len(tape)) < 0.4
    pick[:4] = True  # the arguments have many users
    tape["opcode_uses"] = np.where(pick, (ou & 0xFFFF0000) | 1, ou)
    p = api.default_params(localsubdiv=5, pruning=0, normal_viz=1)
    gs, os_ = Scene(device, Tape.upload(device, tape), p), oracle.Scene(tape, p)
    for time in TIMES:
        gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())


@pytest.mark.gpu
@pytest.mark.parametrize("parents", [1, 2, 4])
def test_directed_narrow_equals_wide(device, parents):
    """Outward rounding: the same octree from the one-warp interpreter alone,
    without pruning, and from the block-wide one."""
    tape = mixed_tape(300, 7)
    p = dict(localsubdiv=6, delta=0.02, rounding_mode=1)
    ref = None
    for threshold, pruning in ((0xFFFFFFFF, 1), (0xFFFFFFFF, 0), (1, 1)):
        t = Tape.upload(device, tape)
        t.narrow_parents = parents
        t.wide_threshold = threshold
        s = Scene(device, t, api.default_params(pruning=pruning, **p))
        cells = []
        for time in TIMES:
            s.invert(time)
            cells.append(s.cells())
        if ref is None:
            ref = cells
        else:
            for a, b in zip(cells, ref):
                assert_cells_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("live", [103, 104, 107])
def test_widest_register_files_run(device, live):
    """Tapes of 104, 105 and 108 registers: the largest register files that eight
    warps of a block hold beside their instruction buffers."""
    b = scenes.IRBuilder()
    r = b.sub(b.sqrt(b.add(b.add(b.mul(b.X, b.X), b.mul(b.Y, b.Y)), b.mul(b.Z, b.Z))), 1.5)
    v = [b.add(b.mul(b.X if i % 2 else b.Y, 0.01 * i), 2.0) for i in range(live - 1)]
    acc = r
    for x in reversed(v):
        acc = b.min(acc, b.add(x, b.T))
    tape = api.IR.new(b.text(acc)).gpu_instructions
    t = Tape.upload(device, tape)
    assert t.registers == live + 1
    p = api.default_params(localsubdiv=4, pruning=0)
    gs, os_ = Scene(device, t, p), oracle.Scene(tape, p)
    for time in TIMES[:2]:
        gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())


@pytest.mark.gpu
@pytest.mark.parametrize("scene", ["csg", "division"])
def test_directed_infinite_sensitivities_match_full_tape(device, scene):
    """Cells around roots at zero below decided maxima (distances to boxes), on
    a tape whose rules are finite but for the roots' and on one with
    quotients: pruned tapes give what the full tape gives, on one warp and
    block-wide, bit for bit."""
    if scene == "csg":
        tape = api.IR.new(scenes.csg(24, 3)).gpu_instructions
    else:
        b = scenes.IRBuilder()
        acc = b.sub(b.sqrt(b.add(b.mul(b.X, b.X), b.mul(b.Y, b.Y))), 0.9)
        for i in range(14):
            q = b.max(b.sub(b.abs(b.sub(b.X, 0.2 * i - 1.4)), 0.08), 0.0)
            r = b.max(b.sub(b.abs(b.add(b.Z, b.mul(b.T, 0.3))), 0.2), 0.0)
            s = b.sub(b.sqrt(b.add(b.mul(q, q), b.mul(r, r))), 0.03)
            acc = b.min(acc, b.max(b.div(s, 3.0), b.sub(b.Y, 0.5)))
        tape = api.IR.new(b.text(acc)).gpu_instructions
    ref = None
    for threshold, pruning in ((0xFFFFFFFF, 0), (0xFFFFFFFF, 1), (1, 1)):
        t = Tape.upload(device, tape)
        t.wide_threshold = threshold
        s = Scene(device, t, api.default_params(localsubdiv=6, delta=0.01, rounding_mode=1, normal_viz=1, pruning=pruning))
        cells = []
        for time in TIMES:
            s.invert(time)
            cells.append(s.cells())
        if ref is None:
            ref = cells
        else:
            for a, c in zip(cells, ref):
                assert_cells_equal(a, c)


def argument_tape(arg: str, kind: str) -> np.ndarray:
    """Moving spheres, less a little of an argument beyond the clamp of `fix`
    which a min/max that is always decided passes on: its last use, so the
    copy that it becomes when pruned goes to the argument's own register."""
    b = scenes.IRBuilder()
    acc = None
    for i in range(30):
        c = [0.9 * np.cos(i), 0.9 * np.sin(2.0 * i), 0.9 * np.sin(i)]
        d = [b.sub(v, float(ck)) for v, ck in zip((b.Y, b.Z), c)]
        s = b.sub(b.sqrt(b.add(b.mul(d[0], d[0]), b.mul(d[1], d[1]))), 0.3 + 0.01 * i)
        s = b.add(s, 0.0)
        acc = s if acc is None else b.min(acc, s)
    v = b.T if arg == "t" else b.X
    m = b.min(v, 2.0e6) if kind == "literal" else b.max(b.min(b.mul(b.Y, 0.1), 3.0), v)
    acc = b.sub(acc, b.mul(m, 2.0e-7))
    return api.IR.new(b.text(acc)).gpu_instructions


@pytest.mark.gpu
@pytest.mark.parametrize("threshold", [0xFFFFFFFF, 100])
@pytest.mark.parametrize("kind", ["literal", "register"])
@pytest.mark.parametrize("arg", ["t", "x"])
def test_copies_of_arguments_beyond_the_clamp_are_kept(device, arg, kind, threshold):
    """`fix` clamps what a min/max passes on; the four arguments are as given.
    A pruned tape has to clamp the argument where the full tape does."""
    tape = argument_tape(arg, kind)
    assert len(tape) >= 260  # a bundled form
    p = dict(localsubdiv=5, delta=0.02)
    if arg == "x":
        p.update(root_lo=(1.4e6, -2.0, -2.0), root_hi=(1.4e6 + 4.0, 2.0, 2.0))
    p = api.default_params(**p)
    t = Tape.upload(device, tape)
    t.wide_threshold = threshold
    gs, os_ = Scene(device, t, p), oracle.Scene(tape, p)
    for time in ([1.4e6, 1.4e6 + 1.0] if arg == "t" else TIMES[:2]):
        gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())
