"""Lists of boxes by the one-warp and the block-wide interpreter: counts that
end on, before and after a warp's boxes, tapes with and without a bundled
form, the widest register file, infinite and NaN bounds, and both routes on
the same boxes."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from temporalsetinversion_b200 import Tape, api, scenes
from test_gpu_narrow import mixed_tape
from test_gpu_ops import random_boxes

MANY = 20000  # boxes enough for one warp per 32 of them to be the faster way


def many_registers(live: int) -> np.ndarray:
    b = scenes.IRBuilder()
    v = [b.add(b.mul(b.X if i % 2 else b.Y, 0.01 * i), 2.0) for i in range(live)]
    acc = b.sub(b.Z, b.T)
    for x in reversed(v):
        acc = b.min(acc, b.add(x, b.T))
    return api.IR.new(b.text(acc)).gpu_instructions


TAPES = {
    "one": lambda: api.IR.new(scenes.IRBuilder().text("%0")).gpu_instructions,  # no instruction at all
    "short": lambda: mixed_tape(40, 3),
    "long": lambda: mixed_tape(300, 4),
    "registers_255": lambda: many_registers(253),
    "registers_256": lambda: many_registers(254),
}


def boxes_of(n: int, seed: int) -> np.ndarray:
    b = random_boxes(max(n, 64), np.random.default_rng(seed))[:n]
    wild = [(-np.inf, np.inf), (1e30, np.inf), (-np.inf, -3.0), (np.nan, np.nan), (-2e6, 3e6)]
    for k, (lo, hi) in enumerate(wild):
        if n > 8 * (k + 1):
            b[8 * (k + 1), 2 * (k % 4):2 * (k % 4) + 2] = lo, hi
    return b


def same(a: np.ndarray, b: np.ndarray) -> bool:
    return bool(((a == b) | (np.isnan(a) & np.isnan(b))).all())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 70, MANY])
@pytest.mark.parametrize("name", sorted(TAPES))
def test_boxes_match_oracle(device, name, n):
    tape = TAPES[name]()
    boxes = boxes_of(n, n)
    t = Tape.upload(device, tape)
    if name.startswith("registers"):
        assert t.registers == int(name[-3:])
    for reverse in (True, False):
        assert same(t.eval_boxes(boxes, reverse=reverse), oracle.eval_boxes(tape, boxes, reverse=reverse))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["short", "long"])
def test_directed_boxes_do_not_depend_on_the_route(device, name):
    tape = TAPES[name]()
    boxes = boxes_of(MANY, 5)
    t = Tape.upload(device, tape)
    all_ = t.eval_boxes(boxes, rounding_mode=1)
    for n in (1, 33, 70):
        assert same(t.eval_boxes(boxes[:n], rounding_mode=1), all_[:n])


@pytest.mark.gpu
def test_sqrt_at_the_edges_of_its_short_form(device):
    """Zeros of both signs, negative lower bounds, the ends of the range of
    the branch-free root and beyond them, denormals, infinities and NaN."""
    b = scenes.IRBuilder()
    tape = api.IR.new(b.text(b.sqrt("%0"))).gpu_instructions
    f = np.float32
    edge = [0.0, -0.0, -1.0, 1e-45, 1e-38, np.nextafter(f(1e-23), f(0)), 1e-23, np.nextafter(f(1e-23), f(1)), 1e-9,
            0.25, 2.0, 3.0, np.nextafter(f(1e23), f(0)), 1e23, np.nextafter(f(1e23), f(np.inf)), 3e38, np.inf, -np.inf,
            np.nan]
    pairs = np.array([(x, y) for x in edge for y in edge], np.float32)
    rng = np.random.default_rng(1)
    more = np.sort((rng.uniform(1, 4, (4000, 2)) * 2.0 ** rng.integers(-84, 84, (4000, 1))).astype(np.float32), axis=1)
    pairs = np.concatenate([pairs, more])
    boxes = np.zeros((len(pairs), 8), np.float32)
    boxes[:, 0:2] = pairs
    t = Tape.upload(device, tape)
    assert same(t.eval_boxes(boxes), oracle.eval_boxes(tape, boxes))
