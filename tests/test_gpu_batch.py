"""Batched form: many scenes (different tapes, depths, times) in one fused
launch sequence give exactly what each gives alone."""
from __future__ import annotations

import math

import numpy as np
import pytest

from conftest import assert_cells_equal
from temporalsetinversion_b200 import Scene, Tape, _native as N, api, scenes


def _make(device, specs):
    out = []
    for text, L in specs:
        tape = Tape.from_llvm_ir(device, text)
        out.append(Scene(device, tape, api.default_params(localsubdiv=L)))
    return out


SPECS = [(scenes.csg(16, 1, 0.9), 6), (scenes.spheres16(2), 7), (scenes.csg(40, 3, 0.9), 5), (scenes.swept(6, 5), 6)]


@pytest.mark.gpu
def test_batch_equals_alone(device):
    alone = _make(device, SPECS)
    mixed = _make(device, SPECS)
    times = [[0.0, 0.1, 0.3], [0.2, 0.25, 0.3], [0.9, 0.5, 0.1], [0.0, 1 / 60, 2 / 60]]
    cam = scenes.camera_look_at((0.4, 0.8, 2.4))
    for f in range(3):
        reqs = []
        for i, s in enumerate(mixed):
            u = api.make_uniforms(cam, (96, 64), times[i][f])
            reqs.append((s, times[i][f], math.nan, u))
        res = api.run_batch(device, reqs)
        for i, s in enumerate(alone):
            st = s.invert(times[i][f])
            u = api.make_uniforms(cam, (96, 64), times[i][f])
            img = s.trace(u)
            assert res[i]["stats"].error_flags == 0
            assert_cells_equal(mixed[i].cells(), s.cells())
            assert np.array_equal(res[i]["depth"], img["depth"])
            assert np.array_equal(res[i]["rgba"], img["rgba"])


@pytest.mark.gpu
def test_graph_replays_equal_plain_frames(device):
    """A captured batch replayed over several frames (new times and cameras
    each launch) gives the plain path's octrees and images."""
    alone = _make(device, SPECS[:3])
    graphed = _make(device, SPECS[:3])
    res = (96, 64)
    eyes = [(0.4, 0.8, 2.4), (0.5, 0.7, 2.3), (0.6, 0.6, 2.2)]
    times = [[0.0, 0.2, 0.9], [0.05, 0.25, 0.8], [0.1, 0.3, 0.7]]
    reqs = [(s, times[0][i], math.nan, api.make_uniforms(scenes.camera_look_at(eyes[0]), res, times[0][i]))
            for i, s in enumerate(graphed)]
    g = api.BatchGraph(device, reqs)
    try:
        for f in range(3):
            unis = [api.make_uniforms(scenes.camera_look_at(eyes[f]), res, times[f][i]) for i in range(3)]
            g.launch(times[f], unis)
            st = g.wait()
            assert st.error_flags == 0 and st.device_ms > 0.0 and st.cells_evaluated > 0
            for i, s in enumerate(alone):
                s.invert(times[f][i])
                want = s.trace(unis[i])
                got = graphed[i].image(*res)
                assert_cells_equal(graphed[i].cells(), s.cells())
                assert np.array_equal(got["depth"], want["depth"])
                assert np.array_equal(got["rgba"], want["rgba"])
    finally:
        g.close()


@pytest.mark.gpu
def test_graph_survives_a_larger_scratch():
    """A graph whose cells live in the context's global scratch replays after a
    scene with larger cells has had that scratch replaced."""
    from temporalsetinversion_b200 import Device

    dev = Device()
    try:
        p = api.default_params(localsubdiv=3, delta=0.02)
        small = Tape.from_llvm_ir(dev, scenes.csg(700, 2))
        a, b = Scene(dev, small, p), Scene(dev, small, p)
        g = api.BatchGraph(dev, [(a, 0.0, float("nan"), None)])
        big = Tape.from_llvm_ir(dev, scenes.csg(1400, 2))
        c = Scene(dev, big, p)
        c.invert(0.0)
        for t in (0.0, 0.05):
            g.launch([t])
            g.wait()
            b.invert(t)
            assert_cells_equal(a.cells(), b.cells())
        g.close()
    finally:
        dev.close()


@pytest.mark.gpu
def test_graph_reads_its_own_rows_after_a_wider_batch():
    """A graph's counters and error status after a batch of more scenes than
    the context had readback rows for, which makes the context take others."""
    from temporalsetinversion_b200 import Device

    with Device() as dev:
        p = api.default_params(localsubdiv=4, delta=0.02)
        tape = Tape.from_llvm_ir(dev, scenes.spheres16(0))
        a, b = Scene(dev, tape, p, 1 << 14), Scene(dev, tape, p, 1 << 14)
        full = Scene(dev, tape, p, 64)  # a pool of a few bricks: the first frame exhausts it
        good = api.BatchGraph(dev, [(a, 0.0, math.nan, None)])
        bad = api.BatchGraph(dev, [(full, 0.0, math.nan, None)])
        flat = api.default_params(localsubdiv=1)
        api.run_batch(dev, [(Scene(dev, tape, flat, 1 << 10), 0.0, math.nan, None) for _ in range(130)])
        for t in (0.0, 0.05):
            good.launch([t])
            st, want = good.wait(), b.invert(t)
            assert st.cells_evaluated == want.cells_evaluated > 0 and st.error_flags == 0
            assert_cells_equal(a.cells(), b.cells())
        bad.launch([0.0])
        with pytest.raises(N.TsiError) as e:
            bad.wait()
        assert e.value.status == 4  # TSI_ERR_OOM
        good.close()
        bad.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 5, 65])
def test_frames_of_one_launch_equal_their_own(device, n):
    """Frames traced together: sizes that are no multiple of a block's tile,
    down to one pixel, field normals and path tracing among them, and one more
    scene than a launch takes."""
    sizes = [(96, 64), (33, 17), (1, 1), (17, 9), (64, 8)]
    kinds = [dict(), dict(fast_normals=1), dict(cinematic=1, samples=2), dict(normal_viz=1), dict()]
    texts = [scenes.csg(16, 1, 0.9), scenes.spheres16(2)]
    tapes = [Tape.from_llvm_ir(device, t) for t in texts]
    cam = scenes.camera_look_at((0.4, 0.8, 2.4))
    reqs, alone = [], []
    for i in range(n):
        p = api.default_params(localsubdiv=4 + i % 2, **kinds[i % 5])
        u = api.make_uniforms(cam, sizes[i % 5], 0.1)
        reqs.append((Scene(device, tapes[i % 2], p, 1 << 14), 0.1, math.nan, u))
        if i < 10 or i == n - 1:
            s = Scene(device, tapes[i % 2], p, 1 << 14)
            s.invert(0.1)
            alone.append((i, s.trace(u)))
    res = api.run_batch(device, reqs)
    for i, img in alone:
        for k in ("depth", "rgba", "normal"):
            assert np.array_equal(res[i][k], img[k], equal_nan=True)
