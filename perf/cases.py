"""The work a user of the framework has it do, as cases that can be timed and
whose outputs can be compared: clips of animated scenes (inversion and trace
per frame), camera flights over a resident octree, swept volumes, rigorous
(directed) inversion, path-traced frames, batches replayed as a CUDA graph,
one animation split over subtree scenes, and interval evaluation of a tape on
lists of boxes.  Scene generators, tape sizes, levels, resolutions and options
are those of the benchmark and the tests; every call is a public entry point.

A clip starts from the root (Scene.reset: the program's first_eval) and
carries its octree over from frame to frame, so one pass holds the first
frame and the temporally reused ones, and every pass gives the same outputs.
Frames stay on the device, as a compositor, encoder or viewer on the GPU reads
them, except in the streamed clip, whose frames go to pinned host memory.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from temporalsetinversion_b200 import IR, Device, Scene, Tape, _native as N, api, scenes, split

NAN = math.nan
_device = None


def _dev() -> Device:
    """A program keeps one device context for all of its scenes."""
    global _device
    if _device is None:
        _device = Device(0)
    return _device


# ------------------------------------------------------------------ the cases
def _clip(name, scene, prims, level, width, height, frames, **kw):
    case = {"name": name, "kind": "clip", "scene": scene, "prims": prims, "level": level, "width": width,
            "height": height, "frames": frames, "directed": False, "fast_normals": False, "stream": False}
    case.update(kw)
    return case


def listed():
    return [
        # one frame of the small plain configuration from scratch, with the
        # finite-difference normals the reference's own parameters enable:
        # the smallest call, launches and latency count
        _clip("still_spheres16_L8_360p", "spheres", 16, 8, 640, 360, 1, fast_normals=True),
        # the headline animation: 256 primitives, localsubdiv 10, 1080p,
        # synchronous plain calls frame after frame
        _clip("clip_csg256_L10_1080p", "csg", 256, 10, 1920, 1080, 6),
        # the same animation end to end: frames queued without host waits,
        # each frame's pixels copied to pinned host memory
        _clip("stream_csg256_L10_1080p", "csg", 256, 10, 1920, 1080, 4, stream=True),
        # a long tape (about 18 thousand instructions), square preview frames
        _clip("clip_csg1024_L9_512", "csg", 1024, 9, 512, 512, 3),
        # swept volumes of rotating, shrinking primitives (sines, cosines,
        # an exponential), sub-step after sub-step
        _clip("swept64_L9_720p", "swept", 64, 9, 1280, 720, 4),
        # rigorous bounds: outward rounding, a mid-size scene
        _clip("directed_csg64_L8_720p", "csg", 64, 8, 1280, 720, 3, directed=True),
        # a viewer flying around a still scene: the octree is resident, every
        # frame is a trace from another camera
        {"name": "orbit_csg256_L9_1440p", "kind": "orbit", "scene": "csg", "prims": 256, "level": 9, "width": 2560,
         "height": 1440, "frames": 4, "cinematic": False, "samples": 1},
        # path-traced stills of the small scene, 8 samples per pixel
        {"name": "cinematic_spheres16_L8_360p", "kind": "orbit", "scene": "spheres", "prims": 16, "level": 8,
         "width": 640, "height": 360, "frames": 1, "cinematic": True, "samples": 8},
        # scenes of uneven tapes and depths, one CUDA-graph replay per step
        {"name": "batch12_512", "kind": "batch", "scenes": 12, "max_prims": 512, "width": 512, "height": 512,
         "frames": 2},
        # one animation cut at the root into eight subtree scenes, composited
        {"name": "split8_csg64_L9_720p", "kind": "split", "prims": 64, "level": 9, "width": 1280, "height": 720,
         "frames": 2},
        # field bounds of a few hundred boxes (a collision query), and field
        # bounds with sensitivities of many boxes on the headline's tape
        {"name": "boxes_csg64_511", "kind": "boxes", "prims": 64, "boxes": 511, "reverse": False, "directed": False},
        {"name": "boxes_csg256_60k_reverse", "kind": "boxes", "prims": 256, "boxes": 60000, "reverse": True,
         "directed": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["clip", "clip", "clip", "clip", "orbit", "orbit", "batch", "split", "boxes", "boxes"])
    width = _log_int(rng, 160, 1920)
    height = max(90, min(1080, int(width * rng.uniform(0.5, 1.0))))
    if kind == "clip":
        scene = rng.choice(["csg", "csg", "csg", "spheres", "swept"])
        prims = 16 if scene == "spheres" else _log_int(rng, 8, 64 if scene == "swept" else 512)
        level = rng.randint(6, 9 if scene == "swept" or prims > 256 else 10)
        directed = rng.random() < 0.2
        fast = rng.random() < 0.2
        if directed:
            prims, level = min(prims, 96), min(level, 8)
        if fast:
            prims = min(prims, 96)
        return {"kind": "clip", "scene": scene, "prims": prims, "level": level, "width": width, "height": height,
                "frames": rng.randint(1, 4), "directed": directed, "fast_normals": fast,
                "stream": rng.random() < 0.25}
    if kind == "orbit":
        cinematic = rng.random() < 0.4
        if cinematic:
            width, height = min(width, 640), min(height, 360)
        return {"kind": "orbit", "scene": rng.choice(["csg", "spheres"]), "prims": _log_int(rng, 16, 64 if cinematic else 256),
                "level": rng.randint(6, 8 if cinematic else 10), "width": width, "height": height,
                "frames": 1 if cinematic else rng.randint(1, 4), "cinematic": cinematic,
                "samples": rng.choice([1, 3, 8]) if cinematic else 1}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 12), "max_prims": _log_int(rng, 32, 512),
                "width": min(width, 512), "height": min(height, 512), "frames": rng.randint(1, 2)}
    if kind == "split":
        return {"kind": "split", "prims": _log_int(rng, 16, 128), "level": rng.randint(7, 9), "width": min(width, 1280),
                "height": min(height, 720), "frames": rng.randint(1, 2)}
    return {"kind": "boxes", "prims": _log_int(rng, 8, 256), "boxes": _log_int(rng, 1, 60000),
            "reverse": rng.random() < 0.5, "directed": rng.random() < 0.3}


# ------------------------------------------------------------------ scenes
def _text(scene: str, prims: int, seed: int) -> str:
    if scene == "spheres":
        return scenes.spheres16(seed)
    if scene == "swept":
        return scenes.swept(prims, seed)
    return scenes.csg(prims, seed)


# opcodes of the 32-byte instruction layout (tsi.h TSI_OP_*) these scenes use
_ADD, _SUB, _MUL, _EXP, _SQR, _SQRT, _SIN, _COS, _NEG, _MIN, _MAX, _ABS, _RET = 5, 6, 7, 9, 11, 12, 14, 15, 16, 17, 18, 19, 28
_PI, _HALFPI = 3.1415927410125732, 1.5707963705062866  # the f32 constants of the interval rules


def _decode(text: str):
    """(op, operand kinds, left, right, literal) of every instruction, and the
    last instruction that reads each value."""
    g = IR.new(text).gpu_instructions
    ou, lr = g["opcode_uses"].astype(np.int64), g["larg_rarg"].astype(np.int64)
    rows = list(zip(((ou >> 16) & 0x3FFF).tolist(), (ou >> 30).tolist(), (lr >> 16).tolist(), (lr & 0xFFFF).tolist(),
                    g["literal"].astype(np.float64).tolist()))
    last = list(range(len(rows)))
    for j in range(4, len(rows)):
        top, a, b = rows[j][1], rows[j][2], rows[j][3]
        if top in (0, 1):
            last[a] = j
        if top in (0, 2):
            last[b] = j
    return rows, last


def _sin64(lo, hi):
    lq, hq = np.floor(lo / _HALFPI), np.floor(hi / _HALFPI)
    whole = (hi - lo > 2 * _PI) | (hq - lq > 4.0)
    lq, hq = lq - 4.0 * np.floor(lq / 4.0), hq - 4.0 * np.floor(hq / 4.0)
    a, b = np.sin(lo), np.sin(hi)
    mn, mx = np.minimum(a, b), np.maximum(a, b)
    same = lq == hq
    whole |= same & (hi - lo > _PI)
    mono = same | ((lq == 3) & (hq == 0)) | ((lq == 1) & (hq == 2))
    top = ~mono & ((lq == 0) | (lq == 3)) & ((hq == 1) | (hq == 2))
    bot = ~mono & ((lq == 1) | (lq == 2)) & ((hq == 3) | (hq == 0))
    whole |= ~mono & ~top & ~bot
    return np.where(whole | bot, -1.0, mn), np.where(whole | top, 1.0, mx)


def _bounds64(rows, last, args):
    """Interval bounds of the scene's field over boxes, float64: args are four
    (lo, hi) pairs of arrays."""
    vals = {k: v for k, v in enumerate(args)}
    drop = {}
    for v, j in enumerate(last):
        drop.setdefault(j, []).append(v)
    out = None
    with np.errstate(all="ignore"):
        for j in range(4, len(rows)):
            op, top, l, r, lit = rows[j]
            c = (np.float64(lit), np.float64(lit))
            (al, ah) = vals[l] if top in (0, 1) else c
            (bl, bh) = vals[r] if top in (0, 2) else c
            if op == _ADD: v = (al + bl, ah + bh)
            elif op == _SUB: v = (al - bh, ah - bl)
            elif op == _MUL:
                if top == 1: v = (al * bl, ah * bl) if lit >= 0.0 else (ah * bl, al * bl)
                else:
                    p, q, s, t = al * bl, al * bh, ah * bl, ah * bh
                    v = (np.minimum(np.minimum(p, q), np.minimum(s, t)), np.maximum(np.maximum(p, q), np.maximum(s, t)))
            elif op == _SQR:
                p, q = al * al, ah * ah
                z = (al <= 0.0) & (ah >= 0.0)
                v = (np.where(z, 0.0, np.minimum(p, q)), np.maximum(p, q))
            elif op == _SQRT: v = (np.sqrt(np.maximum(al, 0.0)), np.sqrt(np.maximum(ah, 0.0)))
            elif op == _EXP: v = (np.exp(al), np.exp(ah))
            elif op == _SIN: v = _sin64(al, ah)
            elif op == _COS: v = _sin64(al + _HALFPI, ah + _HALFPI)
            elif op == _NEG: v = (-ah, -al)
            elif op == _ABS:
                z = (al <= 0.0) & (ah >= 0.0)
                n = ah < 0.0
                v = (np.where(z, 0.0, np.where(n, -ah, al)), np.where(z, np.maximum(-al, ah), np.where(n, -al, ah)))
            elif op == _MIN: v = (np.minimum(al, bl), np.minimum(ah, bh))
            elif op == _MAX: v = (np.maximum(al, bl), np.maximum(ah, bh))
            elif op == _RET: v = (al, ah)
            else: raise ValueError("opcode %d" % op)
            out = vals[j] = v
            for d in drop.get(j, ()):
                if d != j:
                    vals.pop(d, None)
    return out


def _pick_scene(rng, scene: str, prims: int, time: float) -> str:
    """A scene with something in view: a random tree of unions and
    intersections may be empty, and nobody animates an empty scene."""
    text = ""
    for _ in range(12):
        text = _text(scene, prims, int(rng.integers(1 << 30)))
        rows, last = _decode(text)
        p = rng.uniform(-1.0, 1.0, (3, 1000))
        t = np.full(1000, time)
        f, _ = _bounds64(rows, last, [(p[0], p[0]), (p[1], p[1]), (p[2], p[2]), (t, t)])
        if 0.004 <= float(np.mean(f <= 0.0)) <= 0.6:
            break
    return text


# ------------------------------------------------------------------ state
class _Frame:
    """A scene's frame on the device (tsi_scene_image_device) as a torch tensor
    sees it; it keeps the scene's owner, so the buffers outlive the tensor."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": "<f4", "version": 3}


def _images(st, scene: Scene) -> dict:
    im = N.ImageDevice()
    N.check(scene.device.lib.tsi_scene_image_device(scene.handle, C.byref(im)), "tsi_scene_image_device")
    w, h = im.width, im.height
    return {"rgba": torch.as_tensor(_Frame(im.rgba, (h, w, 4), st), device="cuda"),
            "depth": torch.as_tensor(_Frame(im.depth, (h, w), st), device="cuda"),
            "normal": torch.as_tensor(_Frame(im.normal, (h, w, 3), st), device="cuda")}


_COUNTS = ("parents_expanded", "cells_evaluated", "cells_ambiguous", "cells_empty", "cells_full", "cells_enqueued",
           "cells_reused")


def _counts(stats) -> list:
    return [int(getattr(stats, k)) for k in _COUNTS]


class _State:
    """What a program holds; given back in the order the library wants."""

    def __init__(self, case):
        self.case = case
        self.scenes, self.tapes, self.graph, self.split = [], [], None, None

    def __del__(self):
        try:
            if self.graph is not None:
                self.graph.close()
            if self.split is not None:
                self.split.close()
            for s in self.scenes:
                s.close()
            for t in self.tapes:
                t.close()
        except Exception:
            pass


def _params(case, **kw):
    return api.default_params(localsubdiv=case["level"], delta=0.01, pointsample=1, **kw)


def _capacity(level: int) -> int:
    return (8 << 20) if level >= 9 else (2 << 20)


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 7919])
    dev = _dev()
    st = _State(case)
    kind = case["kind"]
    t0 = float(rng.uniform(0.0, 0.9))
    if kind == "boxes":
        st.text = _pick_scene(rng, "csg", case["prims"], t0)
        st.tapes = [Tape.from_llvm_ir(dev, st.text)]
        n = case["boxes"]
        c = rng.uniform(-1.0, 1.0, (n, 3))
        h = 2.0 ** rng.uniform(-10.0, -3.0, (n, 1))
        dt = np.where(rng.uniform(size=n) < 0.5, 0.0, 1.0 / 60.0)
        t = rng.uniform(0.0, 1.0, n)
        b = np.empty((n, 8), np.float32)
        b[:, 0:6:2], b[:, 1:6:2] = c - h, c + h
        b[:, 6], b[:, 7] = t, t + dt
        st.boxes = b
        return st
    w, hgt = case["width"], case["height"]
    if kind == "batch":
        reqs = []
        for _ in range(case["scenes"]):
            n = int(round(math.exp(rng.uniform(math.log(8), math.log(case["max_prims"])))))
            level = int(rng.integers(7, 10))
            ti = float(rng.uniform(0.0, 0.9))
            tape = Tape.from_llvm_ir(dev, _pick_scene(rng, "csg", n, ti))
            sc = Scene(dev, tape, api.default_params(localsubdiv=level, delta=0.01, pointsample=1, lipschitz_corrected=1),
                       _capacity(level))
            st.tapes.append(tape)
            st.scenes.append(sc)
            reqs.append((sc, ti, NAN, api.make_uniforms(scenes.camera_on_sphere(rng, 2.5), (w, hgt), ti)))
        st.reqs = reqs
        st.graph = api.BatchGraph(dev, reqs)
        return st
    scene = case.get("scene", "csg")
    text = _pick_scene(rng, scene, case["prims"], t0)
    tape = Tape.from_llvm_ir(dev, text)
    st.tapes.append(tape)
    k = case["frames"]
    st.views = [scenes.camera_on_sphere(rng, 2.5)] * k
    if kind == "split":
        st.split = split.SubtreeSplit(dev, tape, _params(case, lipschitz_corrected=1), 1, voxel_capacity=4 << 20)
        st.times = [t0 + i / 119.0 for i in range(k)]
    elif kind == "orbit":
        p = _params(case, lipschitz_corrected=1)
        if case["cinematic"]:
            p = _params(case, fast_normals=1, cinematic=1, samples=case["samples"], see_background=1)
        sc = Scene(dev, tape, p, _capacity(case["level"]))
        st.scenes.append(sc)
        st.counts = _counts(sc.invert(t0))
        st.times = [t0] * k
        a0 = rng.uniform(0.0, 2.0 * math.pi)
        st.views = [scenes.camera_look_at((2.4 * math.cos(a0 + 0.3 * i), 0.8, 2.4 * math.sin(a0 + 0.3 * i)))
                    for i in range(k)]
    else:
        swept = scene == "swept"
        p = _params(case, swept_volume=int(swept), lipschitz_corrected=0 if swept else 1,
                    fast_normals=int(case["fast_normals"]),
                    rounding_mode=1 if case["directed"] else 0)
        sc = Scene(dev, tape, p, _capacity(case["level"]))
        st.scenes.append(sc)
        st.times = [t0 + i / 119.0 for i in range(k)]
        st.t0s = [t - 1.0 / 64.0 if swept else NAN for t in st.times]
        if case["stream"]:
            st.pinned = [torch.empty((hgt, w, 4), dtype=torch.float32, pin_memory=True) for _ in range(k)]
    st.uniforms = [api.make_uniforms(v, (w, hgt), t) for v, t in zip(st.views, st.times)]
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "boxes":
        out = st.tapes[0].eval_boxes(st.boxes, rounding_mode=1 if case["directed"] else 0, reverse=case["reverse"])
        return {"field": out[:, :2], "sens": out[:, 2:]} if case["reverse"] else {"field": out[:, :2]}
    if kind == "batch":
        for s in st.scenes:
            s.reset()
        counts = []
        for i in range(case["frames"]):
            times = [r[1] + i / 60.0 for r in st.reqs]
            unis = [r[3] for r in st.reqs]
            for u, t in zip(unis, times):
                u.time = t
            st.graph.launch(times, unis)
            counts.append(_counts(st.graph.wait()))
        return {"counts": np.array(counts, np.int64), "frames": [_images(st, s) for s in st.scenes]}
    if kind == "split":
        st.split.reset()
        counts = []
        for t, u in zip(st.times, st.uniforms):
            fb, stats = st.split.frame(t, u)
            counts += [_counts(s) for s in stats]
        return {"counts": np.array(counts, np.int64), "rgba": fb["rgba"], "depth": fb["depth"],
                "normal": fb["normal"], "key": fb["key"]}
    sc = st.scenes[0]
    if kind == "orbit":
        for u in st.uniforms:
            sc.trace(u, rgba=False, depth=False, normal=False)  # the frame stays on the device
        return {"counts": np.array(st.counts, np.int64), **_images(st, sc)}
    sc.reset()
    if case["stream"]:
        for t, t0, u, px in zip(st.times, st.t0s, st.uniforms, st.pinned):
            sc.invert_async(t, t0)
            sc.trace_async(u, px.numpy())
        counts = _counts(sc.invert_wait())
        sc.trace_wait()
        return {"counts": np.array(counts, np.int64), "frames": st.pinned}
    counts = []
    for t, t0, u in zip(st.times, st.t0s, st.uniforms):
        counts.append(_counts(sc.invert(t, t0)))
        sc.trace(u, rgba=False, depth=False, normal=False)
    return {"counts": np.array(counts, np.int64), **_images(st, sc)}


# ------------------------------------------------------------------ work
def _cells(level: int) -> float:
    """Cells one inversion evaluates, near enough (measured 0.08 to 0.3 of
    4^level on these scenes)."""
    return 0.1 * 4.0 ** level


def _inversion(level: int) -> dict:
    # a cell: about forty instructions survive pruning, forward and reverse,
    # some eight operations each way; its state read and written once
    n = _cells(level)
    return {"bytes": n * 120.0, "flops": n * 40 * 16.0}


def work(case):
    kind = case["kind"]
    if kind == "boxes":
        n = 18.5 * case["prims"]  # instructions of the tape
        return {"bytes": case["boxes"] * (72.0 if case["reverse"] else 40.0) + 8 * n,
                "flops": case["boxes"] * n * (12.0 if case["reverse"] else 5.0)}
    px = case["width"] * case["height"]
    frame = {"bytes": px * 32.0, "flops": px * 600.0}  # outputs once; some 26 nodes a ray
    k = case["frames"]
    if kind == "batch":
        inv = _inversion(8)
        return {q: k * case["scenes"] * (frame[q] + inv[q]) for q in frame}
    if kind == "orbit":
        mul = 3 * case["samples"] if case["cinematic"] else 1
        return {"bytes": k * frame["bytes"] + _cells(case["level"]) * 60.0, "flops": k * mul * frame["flops"]}
    inv = _inversion(case["level"])
    if kind == "split":
        return {"bytes": k * (px * 40.0 + inv["bytes"]), "flops": k * (8 * frame["flops"] + inv["flops"])}
    mul = 16.0 if case["stream"] else 32.0
    return {"bytes": k * (px * mul + inv["bytes"]), "flops": k * (frame["flops"] + inv["flops"])}


# ------------------------------------------------------------------ 64 bits
def exact(case, seed):
    """The field bounds of the boxes in float64.  An octree and its images
    are f32 constructions (cell boxes, carried-over decisions, a march in
    steps of 1e-4) that have no other value, and sensitivities jump where a
    min/max changes its decision: None for those."""
    if case["kind"] != "boxes" or case["directed"]:
        return None
    st = prepare(case, seed)
    rows, last = _decode(st.text)
    b = st.boxes.astype(np.float64)
    out = np.empty((len(b), 2))
    for i in range(0, len(b), 4096):
        c = b[i:i + 4096]
        lo, hi = _bounds64(rows, last, [(c[:, 2 * q], c[:, 2 * q + 1]) for q in range(4)])
        out[i:i + 4096, 0], out[i:i + 4096, 1] = lo, hi
    return {"field": out, "sens": None} if case["reverse"] else {"field": out}
