"""Octree ray tracing on the GPU against the oracle's restatement of
compute.wgsl `trace` / `rt_main`: depth, normal and colour images bit for
bit, with stored and finite-difference normals, normal visualisation, the
per-scene cameras, render mode and asynchronous read-back."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from golden.make_golden import load_tape
from temporalsetinversion_b200 import Scene, Tape, api, scenes

def _compare(g, o):
    bad = [k for k in ("depth", "normal", "rgba") if g[k].tobytes() != o[k].tobytes()]
    assert not bad, "images differ: %s" % {k: int((g[k] != o[k]).sum()) for k in bad}


@pytest.mark.gpu
@pytest.mark.parametrize("name,src,params,eye", [
    ("spheres16", "spheres16", dict(localsubdiv=7, pointsample=0), (0.3, 0.6, 2.5)),
    ("csg48", "csg48", dict(localsubdiv=7), (-1.5, 1.0, 2.0)),
    ("sponza", "sponza", dict(localsubdiv=6, normal_viz=1), (0.0, 0.0, 8.0)),
    # normals by finite differences of the tape (compute.wgsl:4143-4184 for any scene)
    ("sponza_fast", "sponza", dict(localsubdiv=6, normal_viz=1, fast_normals=1), (0.0, 0.0, 8.0)),
    ("spheres16_fast", "spheres16", dict(localsubdiv=7, pointsample=0, normal_viz=1, fast_normals=1),
     (0.3, 0.6, 2.5)),
])
def test_trace_matches_oracle(device, name, src, params, eye):
    if src == "spheres16":
        tape = api.IR.new(scenes.spheres16(0)).gpu_instructions
    elif src == "csg48":
        tape = api.IR.new(scenes.csg(48, 4)).gpu_instructions
    else:
        tape = load_tape(src)
    p = api.default_params(**params)
    gs = Scene(device, Tape.upload(device, tape), p)
    os_ = oracle.Scene(tape, p)
    times = [0.0, 1 / 60, 2 / 60]
    for t in times:
        gs.invert(t)
        os_.invert(t)
    u = api.make_uniforms(scenes.camera_look_at(eye), (160, 90), times[-1])
    g = gs.trace(u)
    o = os_.trace(u)
    assert (o["depth"] >= 0).sum() > 100, "camera sees the surface"
    _compare(g, o)


@pytest.mark.gpu
def test_trace_scene_offsets(device):
    """scene ids 0/3/4/5 apply rt_main's eye offsets and rotations."""
    tape = load_tape("cradle")
    for sid in (0, 3, 4, 5):
        p = api.default_params(localsubdiv=5, scene_id=sid)
        gs = Scene(device, Tape.upload(device, tape), p)
        os_ = oracle.Scene(tape, p)
        gs.invert(0.0)
        os_.invert(0.0)
        u = api.make_uniforms(scenes.camera_look_at((0.0, 0.0, 0.5), (0.0, 0.0, -1.0)), (64, 48), 0.0)
        _compare(gs.trace(u), os_.trace(u))


@pytest.mark.gpu
def test_rendermode_black(device):
    tape = api.IR.new(scenes.spheres16(0)).gpu_instructions
    gs = Scene(device, Tape.upload(device, tape), api.default_params(localsubdiv=5))
    gs.invert(0.0)
    u = api.make_uniforms(scenes.camera_look_at((0, 0, 2.5)), (32, 32), 0.0, rendermode=1.0)
    g = gs.trace(u)
    assert np.all(g["rgba"] == 0) and np.all(g["depth"] == -1)


@pytest.mark.gpu
def test_trace_async_matches_trace(device):
    """Frames read back asynchronously (pinned buffers, copies overlapping
    the next inversion) equal the synchronous trace's frames."""
    import torch

    text = scenes.csg(24, 5, 0.8)
    params = api.default_params(localsubdiv=6)
    a = Scene(device, Tape.from_llvm_ir(device, text), params)
    b = Scene(device, Tape.from_llvm_ir(device, text), params)
    cam = scenes.camera_look_at((0.5, 0.9, 2.3))
    res = (160, 96)
    bufs = [torch.empty((res[1], res[0], 4), dtype=torch.float32, pin_memory=True) for _ in range(4)]
    want = []
    for f in range(4):
        t = f / 60.0
        u = api.make_uniforms(cam, res, t)
        a.invert(t)
        a.trace_async(u, bufs[f].numpy())
        b.invert(t)
        want.append(b.trace(u, depth=False, normal=False)["rgba"])
    a.trace_wait()
    for f in range(4):
        assert np.array_equal(bufs[f].numpy(), want[f])


@pytest.mark.gpu
def test_pipelined_frames_match_sequential(device):
    """Inversions and traces queued back to back without waiting (frame i's
    copy to host memory overlapping the inversion of frame i + 1) give the
    frames of the sequential invert-then-trace loop: colour, depth and
    normal."""
    import torch

    text = scenes.csg(64, 5, 0.85)
    params = api.default_params(localsubdiv=7)
    a = Scene(device, Tape.from_llvm_ir(device, text), params)
    b = Scene(device, Tape.from_llvm_ir(device, text), params)
    cam = scenes.camera_look_at((0.5, 0.9, 2.3))
    res = (192, 108)
    n = 8
    pin = lambda c: torch.empty((res[1], res[0], c), dtype=torch.float32, pin_memory=True)
    bufs = [(pin(4), pin(1), pin(3)) for _ in range(n)]
    for f in range(n):
        t = f / 30.0
        a.invert_async(t)
        a.trace_async(api.make_uniforms(cam, res, t), *(x.numpy() for x in bufs[f]))
    a.invert_wait()
    a.trace_wait()
    for f in range(n):
        t = f / 30.0
        b.invert(t)
        want = b.trace(api.make_uniforms(cam, res, t))
        rgba, depth, normal = (x.numpy() for x in bufs[f])
        assert np.array_equal(rgba, want["rgba"]), f
        assert np.array_equal(depth.reshape(want["depth"].shape), want["depth"]), f
        assert np.array_equal(normal.reshape(want["normal"].shape), want["normal"]), f



def _steps(lo: float, n: int) -> float:
    return n * float(np.spacing(np.float32(abs(lo))))


@pytest.mark.gpu
@pytest.mark.parametrize("lo,extent", [
    (0.0, 1.0), (0.0, 2.0 ** -18), (0.0, 2.0 ** -19), (1.0e5, _steps(1.0e5, 4)), (1.0e5, _steps(1.0e5, 6)),
    (-1.0e5, _steps(1.0e5, 12)), (1.0e5, _steps(1.0e5, 100)), (1.0e5, _steps(1.0e5, 512))])
def test_walk_at_the_limits_of_ordinary_rays_and_boxes(device, lo, extent):
    """Rays along a diagonal (steps on two and three axes at once) and within
    1e-9 of an axis, boxes of extents around 2^-24, and boxes some steps of
    the numbers at their bounds wide: far from the origin the smallest ones
    round to no extent at all."""
    c = lo + 0.5 * extent
    b = scenes.IRBuilder()
    d = [b.mul(b.sub(b.X, c), 1.0 / extent), b.sub(b.Y, 0.5), b.sub(b.Z, 0.5)]
    s = b.add(b.add(b.mul(d[0], d[0]), b.mul(d[1], d[1])), b.mul(d[2], d[2]))
    tape = api.IR.new(b.text(b.sub(b.sqrt(s), 0.3))).gpu_instructions
    p = api.default_params(localsubdiv=8, root_lo=(lo, 0.0, 0.0), root_hi=(lo + extent, 1.0, 1.0))
    gs, os_ = Scene(device, Tape.upload(device, tape), p), oracle.Scene(tape, p)
    gs.invert(0.0)
    os_.invert(0.0)
    hits = 0
    for eye in ((2.0, 2.0, 2.0), (-2.0, 0.4, 0.6), (3.0, 0.9, 0.2), (1e-9, 0.0, 1.0), (1.0, 1e-7, 1e-9)):
        at = (c + eye[0], 0.5 + eye[1], 0.5 + eye[2])
        u = api.make_uniforms(scenes.camera_look_at(at, (c, 0.5, 0.5)), (33, 33), 0.0)
        g, o = gs.trace(u), os_.trace(u)
        hit = o["depth"] >= 0
        hits += int(hit.sum())
        # (a ray that misses is darkened at every step: what the conversion of
        # an infinity to an integer gives in a box without an extent decides
        # how many it makes, and that differs from the oracle's)
        bare = abs(lo) > 0 and extent < _steps(lo, 32)
        for k in ("depth", "normal", "rgba"):
            eq = g[k].view(np.uint32) == o[k].view(np.uint32)
            assert eq[hit].all() if bare and k == "rgba" else eq.all(), (k, eye)
    assert hits >= 10


@pytest.mark.gpu
@pytest.mark.parametrize("localsubdiv,reaches", [(14, True), (15, False)])
def test_a_ray_of_five_thousand_nodes(device, localsubdiv, reaches):
    """A ray along a sheet thinner than a leaf, between 2048 leaves and twice as
    many, to a ball at its end: the walk stops after 5000 nodes (visits of a
    node and returns to its parent), there as in the oracle."""
    b = scenes.IRBuilder()
    sheet = b.sub(b.abs(b.sub(b.Z, 0.5003)), 1e-5)
    strip = b.sub(b.abs(b.sub(b.X, b.Y)), 0.001)
    d = [b.sub(b.X, 0.97), b.sub(b.Y, 0.97), b.sub(b.Z, 0.5)]
    s = b.add(b.add(b.mul(d[0], d[0]), b.mul(d[1], d[1])), b.mul(d[2], d[2]))
    f = b.min(b.max(sheet, strip), b.sub(b.sqrt(s), 0.05))
    tape = api.IR.new(b.text(f)).gpu_instructions
    p = api.default_params(localsubdiv=localsubdiv, root_lo=(0.0, 0.0, 0.0), root_hi=(1.0, 1.0, 1.0))
    gs, os_ = Scene(device, Tape.upload(device, tape), p), oracle.Scene(tape, p)
    gs.invert(0.0)
    os_.invert(0.0)
    view = scenes.camera_look_at((-0.1, -0.1003, 0.5003), (0.97, 0.97, 0.50035))
    for res in ((1, 1), (5, 5)):
        u = api.make_uniforms(view, res, 0.0)
        g, o = gs.trace(u), os_.trace(u)
        for k in ("depth", "normal", "rgba"):
            assert np.array_equal(g[k].view(np.uint32), o[k].view(np.uint32)), (k, res)
        if res == (1, 1):
            assert (float(o["depth"][0, 0]) >= 0) == reaches and o["visits"] > 3500
