"""The block-wide interpreter at the sizes where it can go wrong: tapes whose
step and min/max counts fall on every remainder of the unroll and of the
packed decision words, every cell on the wide path, its working set in shared
memory and in the global scratch."""
from __future__ import annotations

import pytest

import oracle
from conftest import assert_cells_equal
from temporalsetinversion_b200 import Device, Scene, Tape, api, scenes
from test_gpu_narrow import TIMES, mixed_tape


@pytest.fixture(scope="module")
def scratch_device():
    """A context whose wide cells never fit the shared-memory budget."""
    dev = Device(wide_smem_bytes=1024)
    yield dev
    dev.close()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["shared", "scratch"])
@pytest.mark.parametrize("length", [256, 257, 264, 271, 283, 296, 311, 330])
def test_wide_cells_match_oracle(device, scratch_device, length, where):
    tape = mixed_tape(length, 1000 + length)
    p = api.default_params(localsubdiv=5, delta=0.02, pointsample=length % 2)
    t = Tape.upload(device if where == "shared" else scratch_device, tape)
    t.wide_threshold = 1
    gs, os_ = Scene(t.device, t, p), oracle.Scene(tape, p)
    for time in TIMES:
        gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["shared", "scratch"])
def test_cells_beyond_shared_memory_match_oracle(device, scratch_device, where):
    """Values in the global scratch: with the sensitivities in shared memory
    (the default budget), and with them in the scratch too (no budget, more
    slots than the register files leave room for)."""
    tape = api.IR.new(scenes.csg(1400, 2)).gpu_instructions
    p = api.default_params(localsubdiv=3, delta=0.02)
    t = Tape.upload(device if where == "shared" else scratch_device, tape)
    t.wide_threshold = 1
    gs, os_ = Scene(t.device, t, p), oracle.Scene(tape, p)
    for time in TIMES[:3]:
        gs.invert(time)
        os_.invert(time)
        assert_cells_equal(gs.cells(), os_.cells())


@pytest.mark.gpu
def test_destroyed_tapes_give_their_memory_back(device):
    import torch

    instr = api.IR.new(scenes.csg(64, 5)).gpu_instructions

    def free_after(n):
        for _ in range(n):
            t = Tape.upload(device, instr)
            del t
        return torch.cuda.mem_get_info()[0]

    before = free_after(20)
    # 300 tapes of this scene hold more than 40 MB
    assert before - free_after(300) < 8 << 20
