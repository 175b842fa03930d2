"""Finite-difference normals from the four-point evaluation of the tape where
it can go wrong: register counts around the change from four points a lane to
two and at the largest, every kind of handler, tape lengths around a chunk of
32 instructions, and values beyond the clamp of `fix`, where bounds part."""
from __future__ import annotations

import pytest

import oracle
from temporalsetinversion_b200 import Scene, Tape, api, scenes
from test_gpu_narrow import mixed_tape
from test_gpu_trace import _compare


def ball(b):
    return b.sub(b.sqrt(b.add(b.add(b.mul(b.X, b.X), b.mul(b.Y, b.Y)), b.mul(b.Z, b.Z))), 1.2)


def registers(n: int):
    b = scenes.IRBuilder()
    acc = ball(b)
    v = [b.add(b.mul(b.X if i % 2 else b.Y, 0.01 * i), 5.0) for i in range(n - 2)]
    for x in reversed(v):
        acc = b.min(acc, b.add(x, b.T))
    return api.IR.new(b.text(acc)).gpu_instructions


def clamped():
    """An operand of the last operation leaves the range (and its lower bound
    is not the one chosen near the surface: the normal stays finite)."""
    b = scenes.IRBuilder()
    r = ball(b)
    return api.IR.new(b.text(b.min(r, b.mul(b.mul(b.add(b.abs(r), 1.0), 4.0e9), 2.5e-10)))).gpu_instructions


def rare():
    b = scenes.IRBuilder()
    q = b.div(ball(b), b.add(b.mul(b.X, b.X), 1.5))
    q = b.add(q, b.mul(b.sin(b.mul(b.Y, 3.0)), 0.05))
    q = b.add(q, b.mul(b.exp(b.neg(b.mul(b.X, b.X))), 0.02))
    q = b.sub(q, b.div(0.05, b.add(b.abs(b.Z), 1.0)))
    return api.IR.new(b.text(b.max(q, b.sub(b.Y, 1.0)))).gpu_instructions


TAPES = {
    "registers_26": lambda: registers(26), "registers_27": lambda: registers(27), "registers_96": lambda: registers(96),
    "clamped": clamped, "rare": rare, "len_31": lambda: mixed_tape(31, 2), "len_32": lambda: mixed_tape(32, 2),
    "len_33": lambda: mixed_tape(33, 2), "len_160": lambda: mixed_tape(160, 9),
}


@pytest.mark.gpu
@pytest.mark.parametrize("cinematic", [0, 1])
@pytest.mark.parametrize("name", sorted(TAPES))
def test_fast_normals_match_oracle(device, name, cinematic):
    tape = TAPES[name]()
    t = Tape.upload(device, tape)
    if name.startswith("registers"):
        assert t.registers == int(name[-2:])
    p = api.default_params(localsubdiv=5, pruning=0, fast_normals=1, normal_viz=1 - cinematic, cinematic=cinematic, samples=2,
                           see_background=1)
    gs, os_ = Scene(device, t, p), oracle.Scene(tape, p)
    for time in (0.0, 0.02):
        gs.invert(time)
        os_.invert(time)
    u = api.make_uniforms(scenes.camera_look_at((0.4, 0.8, 4.0)), (72, 41), 0.02)
    o = os_.trace(u)
    assert (o["depth"] >= 0).sum() > 50
    _compare(gs.trace(u), o)
