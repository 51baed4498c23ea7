"""The work that users of this framework have it do, as cases for timing.

Every case goes through the Python binding of the C ABI (virs_b200/capi.py),
the way the scene builders and the benchmark do.  A room is a closed shoebox
of nx x ny x nz voxels with box-shaped furniture standing in it, every
coordinate a whole number of voxels, so that the voxelised room can be
written down without the library.

  calls     the per-step contract of a host that drives every step itself:
            virs_step once per step (upload, one step, read back a sample)
  whole     one whole simulation of a room: start from rest, run, fetch the
            impulse responses
  stretch   a number of steps of a long simulation in progress, with the
            receiver samples of those steps
  batch     the same for many rooms advanced together
  gradient  forward pass with checkpoints and reverse pass: gradients of a
            receiver loss by the absorbers and the source signals
  setup     mesh to classified grid: voxelisation, sponge layer, boundary list
  resample  receiver traces to an audio rate: low-pass cascade with linear
            interpolation, and the windowed-sinc resampler
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from virs_b200 import capi

C0 = 343.0
H = 1.0 / 64.0
STORAGE = {"f32": capi.STORAGE_F32, "f16": capi.STORAGE_F16, "bf16": capi.STORAGE_BF16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # a host in the manner of the reference's own loop: the smallest room, every step a call
        dict(name="calls_tiny_f32", kind="calls", nx=52, ny=44, nz=36, sponge=1, boxes=0, storage="f32", sections=1,
             materials=1, steps=32),
        # a listening room, whole impulse response, a layer of absorbing voxels on every wall
        dict(name="whole_small_f32", kind="whole", nx=160, ny=120, nz=100, sponge=8, boxes=0, storage="f32",
             sections=1, materials=6, steps=2000),
        # a furnished room with a thick sponge layer: more than a third of its voxels are filtered
        dict(name="stretch_furnished_f32", kind="stretch", nx=512, ny=384, nz=192, sponge=16, boxes=20,
             storage="f32", sections=3, materials=4, steps=48, blocking=1, rounding=0),
        # a concert hall, two steps per pass over the fields
        dict(name="stretch_hall_f32", kind="stretch", nx=1024, ny=768, nz=512, sponge=1, boxes=0, storage="f32",
             sections=3, materials=2, steps=48, blocking=2, rounding=0),
        # the same hall in half the memory
        dict(name="stretch_hall_bf16", kind="stretch", nx=1024, ny=768, nz=512, sponge=1, boxes=0, storage="bf16",
             sections=3, materials=2, steps=48, blocking=1, rounding=0),
        # an odd-sized studio in FP16 with stochastic rounding (long runs in 16-bit storage)
        dict(name="stretch_ragged_f16", kind="stretch", nx=701, ny=517, nz=333, sponge=2, boxes=6, storage="f16",
             sections=2, materials=3, steps=48, blocking=1, rounding=1),
        # data generation: rooms of different sizes advanced together
        dict(name="batch_rooms_f32", kind="batch", members=8, side_lo=96, side_hi=256, sponge=1, storage="f32",
             sections=3, materials=3, steps=64),
        # data generation: many small rooms, 16-bit storage
        dict(name="batch_small_bf16", kind="batch", members=24, side_lo=64, side_hi=128, sponge=1, storage="bf16",
             sections=3, materials=2, steps=64),
        # fitting the absorbers of a room to measured responses: one gradient
        dict(name="gradient_room_f32", kind="gradient", nx=128, ny=128, nz=96, sponge=1, boxes=0, storage="f32",
             sections=2, materials=6, steps=256, every=64),
        # loading a furnished room
        dict(name="setup_furnished", kind="setup", nx=320, ny=240, nz=160, sponge=8, boxes=12, materials=4),
        # loading a hall
        dict(name="setup_hall", kind="setup", nx=1024, ny=768, nz=512, sponge=1, boxes=0, materials=4),
        # the end of every simulation: eight traces to 48 kHz
        dict(name="resample_48k", kind="resample", traces=8, steps=4000, rate=48000, lowpass=6, half=245),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, lo, hi):
    """Three extents whose product lies between lo and hi, of different shapes, odd ones among them."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = [rng.uniform(0.6, 1.6) for _ in range(3)]
    s = (v / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
    return dict(zip(("nx", "ny", "nz"), (min(1024, max(28, int(s * f))) for f in a)))


def draw(rng):
    kind = rng.choice(("calls", "whole", "stretch", "stretch", "stretch", "batch", "gradient", "setup", "resample"))
    c = dict(kind=kind, sponge=rng.choice((1, 1, 2, 4, 8)), boxes=rng.choice((0, 4, 12)),
             storage=rng.choice(("f32", "f32", "bf16", "f16")), sections=rng.randint(1, 4), materials=rng.randint(1, 6))
    if kind == "calls":
        c.update(_sizes(rng, 40e3, 2e6), steps=rng.choice((16, 32)), sponge=1, boxes=0, storage="f32", sections=1,
                 materials=1)
    elif kind == "whole":
        c.update(_sizes(rng, 60e3, 2.5e6), steps=_log_int(rng, 300, 1500), boxes=0)
    elif kind == "stretch":
        c.update(_sizes(rng, 2e6, 160e6), steps=_log_int(rng, 24, 48), blocking=rng.choice((1, 1, 2)), rounding=0)
        if c["storage"] != "f32" and rng.random() < 0.4:
            c.update(rounding=1, blocking=1)
    elif kind == "batch":
        lo = rng.randint(48, 96)
        c.update(members=rng.randint(3, 20), side_lo=lo, side_hi=rng.randint(lo + 16, 200), steps=rng.choice((32, 64)),
                 sponge=rng.choice((1, 2)))
        del c["boxes"]
    elif kind == "gradient":
        c.update(_sizes(rng, 60e3, 2.5e6), steps=_log_int(rng, 64, 256), every=rng.choice((16, 32, 64)), storage="f32",
                 boxes=0, sponge=rng.choice((1, 2)))
    elif kind == "setup":
        c.update(_sizes(rng, 500e3, 100e6), materials=rng.randint(3, 6))
        for k in ("storage", "sections"):
            del c[k]
    else:
        c = dict(kind=kind, traces=rng.randint(1, 16), steps=_log_int(rng, 1000, 6000),
                 rate=rng.choice((48000, 44100, 16000)), lowpass=rng.randint(1, 8), half=rng.choice((64, 128, 245)))
    return c


# ---- rooms ------------------------------------------------------------------


def _box(lo, hi, mats):
    """An axis-aligned box, corners in voxels: 8 vertices, 12 triangles, one material per face (-x +x -y +y -z +z)."""
    v = [[(lo, hi)[i][0], (lo, hi)[j][1], (lo, hi)[k][2]] for k in (0, 1) for j in (0, 1) for i in (0, 1)]
    t, m = [], []
    for q, f in zip(((0, 2, 6, 4), (1, 5, 7, 3), (0, 4, 5, 1), (2, 3, 7, 6), (0, 1, 3, 2), (4, 6, 7, 5)), mats):
        t += [[q[0], q[1], q[2]], [q[0], q[2], q[3]]]
        m += [f, f]
    return v, t, m


def _room(c):
    """The boxes of a case's room, fixed by the case: [(lo, hi, face materials)], the shoebox first.  Material
    `materials` is the loudspeaker's (a hard source) where the case has one."""
    n = (c["nx"], c["ny"], c["nz"])
    rng = random.Random("%dx%dx%d" % n)
    m = c["materials"]
    boxes = [((0, 0, 0), n, [k % m for k in range(6)])]
    for _ in range(c.get("boxes", 0)):
        size = [rng.randint(max(3, e // 16), max(4, e // 4)) for e in n]
        lo = [rng.randint(4, e - s - 5) for e, s in zip(n, size)]
        lo[2] = 0
        boxes.append((tuple(lo), tuple(a + s for a, s in zip(lo, size)), [rng.randrange(m)] * 6))
    if c["kind"] == "calls":
        lo = tuple(e // 3 for e in n)
        boxes.append((lo, tuple(a + 2 for a in lo), [m] * 6))
    return boxes


def _mesh(c):
    vs, ts, ms = [], [], []
    for lo, hi, mats in _room(c):
        v, t, m = _box(lo, hi, mats)
        ts += [[i + len(vs) for i in tri] for tri in t]
        vs += v
        ms += m
    return np.array(vs, np.float32) * np.float32(H), np.array(ts, np.uint32), np.array(ms, np.int32)


def _shells(c):
    """Per face of the room's boxes, in order: (slices of the voxels it marks, material).  Voxel k holds the face at
    coordinate k (the last one in each direction also the face at the grid's end)."""
    n = (c["nx"], c["ny"], c["nz"])
    for lo, hi, mats in _room(c):
        a, b = [min(x, e - 1) for x, e in zip(lo, n)], [min(x, e - 1) for x, e in zip(hi, n)]
        for f in range(6):
            s = [slice(a[i], b[i] + 1) for i in range(3)]
            at = (a, b)[f & 1][f >> 1]
            s[f >> 1] = slice(at, at + 1)
            yield tuple(s[::-1]), mats[f]


def _inside_box(c, p, grow=0):
    return any(all(l - grow <= x <= h + grow for x, l, h in zip(p, lo, hi)) for lo, hi, _ in _room(c)[1:])


def _points(c, rng, count, around=None, near=0):
    """Voxels of free air, away from the walls; with `around`, within `near` voxels of it."""
    n = (c["nx"], c["ny"], c["nz"])
    w = c["sponge"]
    got = []
    while len(got) < count:
        lo = [min(w + 2, e // 2 - 1) for e in n]
        hi = [max(e - w - 3, e // 2) for e in n]
        if around is not None:
            lo = [max(a, p - near) for a, p in zip(lo, around)]
            hi = [min(a, p + near) for a, p in zip(hi, around)]
        p = tuple(rng.randint(a, max(a, b)) for a, b in zip(lo, hi))
        if not _inside_box(c, p, 1) and p not in got and p != around:
            got.append(p)
    return got


def _index(c, pts):
    return np.array([(z * c["ny"] + y) * c["nx"] + x for x, y, z in pts], np.uint64)


def _pulses(rng, count, steps):
    """Source signals: a differentiated Gaussian each, of its own width and delay, on a bed of noise."""
    t = np.arange(steps)
    out = []
    for _ in range(count):
        s = rng.uniform(3.0, 8.0)
        u = (t - 3.0 * s) / s
        out.append(rng.uniform(0.5, 2.0) * -u * np.exp(0.5 - 0.5 * u * u))
    noise = np.random.default_rng(rng.randrange(1 << 31)).standard_normal((count, steps))
    return (np.array(out) + 1e-3 * noise).astype(np.float32)


def _absorbers(c, rng):
    """Filter cascades {b0, b1, b2, a1, a2} per material: high-pass first, then peaking cuts (cookbook designs)."""
    fs = math.sqrt(3.0) * C0 / (H * _courant(c))
    out = np.zeros((c["materials"], c["sections"], 5))
    for m in range(c["materials"]):
        for s in range(c["sections"]):
            f = rng.uniform(200.0, 600.0) if s == 0 else rng.uniform(500.0, 6000.0)
            w = 2 * math.pi * f / fs
            if s == 0:
                al, cw = math.sin(w) / (2 * rng.uniform(0.1, 0.7)), math.cos(w)
                b, a = [(1 + cw) / 2, -(1 + cw), (1 + cw) / 2], [1 + al, -2 * cw, 1 - al]
            else:
                al, cw, g = math.sin(w) / (2 * rng.uniform(0.5, 1.5)), math.cos(w), 10 ** (rng.uniform(-12, 0) / 40)
                b, a = [1 + al * g, -2 * cw, 1 - al * g], [1 + al / g, -2 * cw, 1 - al / g]
            out[m, s] = [b[0] / a[0], b[1] / a[0], b[2] / a[0], a[1] / a[0], a[2] / a[0]]
    return out.astype(np.float32)


def _courant(c):
    return 0.5 if c["kind"] == "calls" else 1.0


def _inputs(c, seed):
    """What a pass computes on: positions, signals, absorbers and the pressure at the start."""
    rng = random.Random("%s-%d" % (c["kind"], seed))
    n = min(c["nx"], c["ny"], c["nz"])
    i = dict(coef=_absorbers(c, rng), sphere=None)
    steps = c["steps"]
    if c["kind"] == "calls":
        spk = [lo for lo, _, m in _room(c) if m[0] == c["materials"]][0]
        i["src"], i["sig"] = [], np.zeros((0, steps), np.float32)
        i["rcv"] = _points(c, rng, 1, spk, 6)
        i["hard"] = np.array([rng.uniform(5.0, 12.0) for _ in range(10)], np.float32)
        return i
    i["hard"] = np.zeros(0, np.float32)
    if c["kind"] == "stretch":
        i["src"] = _points(c, rng, 4)
        i["rcv"] = [p for s in i["src"] for p in _points(c, rng, 2, s, 10)]
        r = n // 2 - 2 - c["sponge"]
        i["sphere"] = (c["nx"] // 2, c["ny"] // 2, c["nz"] // 2, r // 2 + rng.randint(0, r // 3), rng.uniform(0.2, 1.0))
    elif c["kind"] == "batch":
        i["src"] = _points(c, rng, 1)
        i["rcv"] = _points(c, rng, 2, i["src"][0], 8)
    else:
        i["src"] = _points(c, rng, 1)
        i["rcv"] = _points(c, rng, 4)
    if c["kind"] == "gradient":
        g = np.random.default_rng(rng.randrange(1 << 31))
        i["loss"] = g.standard_normal((len(i["rcv"]), steps)).astype(np.float32)
        i["rcv"] = _points(c, rng, 4, i["src"][0], 24)
    i["sig"] = _pulses(rng, len(i["src"]), steps)
    return i


def _simulation(c):
    sim = capi.Simulation(capi.default_params(courant=_courant(c), cell_size=H, bbox_nudge=0.0,
                                              sponge_width=c["sponge"], storage=STORAGE[c.get("storage", "f32")],
                                              boundary_form=0 if c["kind"] == "calls" else 1))
    sim.set_material_roles(np.array(list(range(c["materials"])) + [capi.ROLE_SOURCE], np.uint8))
    return sim


def _ready(c, i, reserve):
    sim = _simulation(c)
    sim.set_mesh(*_mesh(c))
    sim.classify()
    sim.set_filters(i["coef"], n_sections=c["sections"])
    sim.set_hard_source(i["hard"] if len(i["hard"]) else np.zeros(1, np.float32))
    if len(i["src"]):
        sim.set_sources(_index(c, i["src"]), i["sig"])
    sim.set_receivers(_index(c, i["rcv"]))
    if c.get("blocking", 1) == 2:
        sim.set_time_blocking(2)
    if c.get("rounding", 0):
        sim.set_rounding(capi.ROUND_STOCHASTIC)
    sim.start(reserve)
    if i["sphere"]:
        sim.init_pressure_sphere(*i["sphere"])
    return sim


def _members(c):
    """The rooms of a batch, fixed by the case."""
    rng = random.Random("%d-%d-%d" % (c["members"], c["side_lo"], c["side_hi"]))
    out = []
    for _ in range(c["members"]):
        side = rng.uniform(c["side_lo"], c["side_hi"])
        a = [rng.uniform(0.7, 1.4) for _ in range(3)]
        g = (a[0] * a[1] * a[2]) ** (1.0 / 3.0)
        out.append(dict(c, **dict(zip(("nx", "ny", "nz"), (max(24, int(side * f / g)) for f in a)))))
    return out


def _sos(c):
    """The cookbook low-pass of a Butterworth cascade below the output rate's band, rows {b0 b1 b2 a0 a1 a2}."""
    fs = math.sqrt(3.0) * C0 / H
    w = 2 * math.pi * 0.42 * min(c["rate"], fs) / fs
    out = []
    for k in range(c["lowpass"]):
        q = 1.0 / (2 * math.cos(math.pi * (2 * k + 1) / (4 * c["lowpass"])))
        al, cw = math.sin(w) / (2 * q), math.cos(w)
        b = (1 - cw) / 2 / (1 + al)
        out.append([b, 2 * b, b, 1.0, -2 * cw / (1 + al), (1 - al) / (1 + al)])
    return np.array(out)


def _trace_case(c):
    """The small room whose responses are resampled."""
    return dict(kind="whole", nx=64, ny=52, nz=44, sponge=2, boxes=0, storage="f32", sections=1, materials=2,
                steps=c["steps"])


def _trace_inputs(c, seed):
    t = _trace_case(c)
    i = _inputs(t, seed)
    i["rcv"] = _points(t, random.Random("traces-%d" % seed), c["traces"])
    return t, i


# ---- a pass -----------------------------------------------------------------


def prepare(case, seed):
    c = case
    k = c["kind"]
    if k == "setup":
        # another seed: other materials on the same surfaces
        rng = random.Random("setup-%d" % seed)
        v, t, m = _mesh(c)
        faces = [rng.randrange(c["materials"]) for _ in range(len(m) // 2)]
        return dict(case=c, verts=v, tris=t, mats=np.repeat(np.array(faces, np.int32), 2))
    if k == "resample":
        t, i = _trace_inputs(c, seed)
        sim = _ready(t, i, c["steps"])
        sim.run(c["steps"])
        sim.synchronize()
        return dict(case=c, sim=sim, sos=_sos(c))
    if k == "batch":
        sims = [_ready(m, _inputs(m, seed * 1000 + j), 1 << 20) for j, m in enumerate(_members(c))]
        return dict(case=c, sims=sims, batch=capi.Batch(sims), done=0)
    i = _inputs(c, seed)
    s = dict(case=c, sim=_ready(c, i, c["steps"] if k in ("whole", "gradient") else 1 << 16), done=0)
    if k == "whole":
        s["sig"] = i["sig"]
        s["out"] = np.zeros((len(i["rcv"]), c["steps"]), np.float32)
    if k == "gradient":
        s["loss"] = i["loss"]
    return s


def run(state):
    c = state["case"]
    k = c["kind"]
    n = c.get("steps", 0)
    if k == "setup":
        sim = _simulation(c)
        sim.set_mesh(state["verts"], state["tris"], state["mats"])
        sim.classify()
        mat, weight = sim.boundary_materials()
        out = dict(index=sim.boundary_indices().view(np.int32), material=mat, weight=weight)
        sim.close()
        return out
    if k == "batch":
        b = state["batch"]
        b.run(n)
        b.synchronize()
        out = [s.ir(state["done"], n) for s in state["sims"]]
        state["done"] += n
        return out
    sim = state["sim"]
    if k == "resample":
        return [sim.postprocess_ir(float(c["rate"]), state["sos"], True),
                sim.postprocess_ir_sinc(float(c["rate"]), half_taps=c["half"])]
    if k == "calls":
        out = [sim.step(state["done"] + j)[1] for j in range(n)]
        state["done"] += n
        return np.array(out, np.float32)
    if k == "whole":
        sim.start(n)
        sim.run_host(n, state["sig"], state["out"])
        return state["out"]
    if k == "gradient":
        sim.forward_checkpointed(n, c["every"])
        ir = sim.ir(0, n)
        gc, gs = sim.adjoint(state["loss"], c["materials"], c["sections"])
        return dict(ir=ir, coef=gc, signal=gs)
    sim.run(n)
    out = sim.ir(state["done"], n)
    state["done"] += n
    return out


# ---- what a pass cannot do without -------------------------------------------


def _step_work(c, steps):
    """Per step: p and p- read, p+ written and a byte of geometry per voxel (with two steps per pass the fields
    once per two steps); per filtered voxel of the room's own layer (the furniture's left out) its states read and written, its
    weight, material and position."""
    v = c["nx"] * c["ny"] * c["nz"]
    e = BYTES[c["storage"]]
    w = c["sponge"]
    n = (c["nx"], c["ny"], c["nz"])
    inner = math.prod(x - 2 for x in n) - math.prod(max(0, x - 2 - 2 * w) for x in n)
    per = (4 * e + 1) / 2 if c.get("blocking", 1) == 2 else 3 * e + 1
    return dict(bytes=steps * (v * per + inner * (2 * 8 * (c["sections"] + 1) + 9)),
                flops=steps * (v * 10.0 + inner * 10.0 * c["sections"]))


def work(case):
    c = case
    k = c["kind"]
    if k == "setup":
        v = c["nx"] * c["ny"] * c["nz"]
        # the flags, materials, codes and normals of every voxel
        return dict(bytes=4.0 * v, flops=0.0)
    if k == "resample":
        fs = math.sqrt(3.0) * C0 / H
        out = c["steps"] * c["rate"] / fs
        return dict(bytes=4.0 * c["traces"] * 2 * (c["steps"] + out),
                    flops=c["traces"] * (9.0 * c["lowpass"] * c["steps"] + 4.0 * c["half"] * out))
    if k == "batch":
        parts = [_step_work(m, c["steps"]) for m in _members(c)]
        return {f: sum(p[f] for p in parts) for f in ("bytes", "flops")}
    w = _step_work(c, c["steps"])
    if k == "gradient":  # forward, forward again, reverse
        w = {f: 3 * x for f, x in w.items()}
    return w


# ---- the same in 64 bits -------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Grid:
    """Flags, boundary voxels and materials of a case's room; the boundary rule is an air voxel within `sponge` of a
    wall voxel, its material that of the nearest one (the first in z, y, x order among equals)."""

    def __init__(self, c, dev):
        shape = (c["nz"], c["ny"], c["nx"])
        wall = torch.zeros(shape, dtype=torch.bool, device=dev)
        mat = torch.zeros(shape, dtype=torch.uint8, device=dev)
        hard = torch.zeros(shape, dtype=torch.bool, device=dev)
        for s, m in _shells(c):
            if m == c["materials"]:
                hard[s], wall[s] = True, False
            else:
                wall[s], hard[s], mat[s] = True, False, m
        w = c["sponge"]
        none = 1 << 30
        key = torch.where(wall, 0, none).to(torch.int32)
        for axis, shift in ((2, 0), (1, 6), (0, 12)):
            best = torch.full(shape, none, dtype=torch.int32, device=dev)
            for d in range(-w, w + 1):
                to = [slice(None)] * 3
                of = [slice(None)] * 3
                to[axis] = slice(max(0, -d), shape[axis] - max(0, d))
                of[axis] = slice(max(0, d), shape[axis] - max(0, -d))
                v = key[tuple(of)]
                v = torch.where(v < none, v + ((d * d << 18) + (d + 32 << shift)), none)
                torch.minimum(best[tuple(to)], v, out=best[tuple(to)])
            key = best
        bnd = (key < none) & ((key >> 18) <= w * w) & ~wall & ~hard
        for axis in range(3):
            for at in (0, shape[axis] - 1):
                s = [slice(None)] * 3
                s[axis] = at
                bnd[tuple(s)] = False
        self.wall, self.hard, self.shape = wall, hard, shape
        self.bnd = torch.nonzero(bnd.reshape(-1)).reshape(-1)
        k = key.reshape(-1)[self.bnd].to(torch.int64)
        step = (shape[1] * shape[2], shape[2], 1)
        near = sum((((k >> s) & 63) - 32) * t for s, t in zip((12, 6, 0), step)) + self.bnd
        self.mat = mat.reshape(-1)[near].to(torch.int64)
        d2 = (k >> 18).to(torch.float64)
        self.weight = ((w + 1 - torch.sqrt(d2)) / w) ** 2
        inner = (slice(1, -1),) * 3
        self.keep = (wall | hard)[inner]
        cnt = torch.zeros(self.keep.shape, dtype=torch.uint8, device=dev)
        for axis in range(3):
            for d in (0, 2):
                s = [slice(1, -1)] * 3
                s[axis] = slice(d, shape[axis] - 2 + d)
                cnt += wall[tuple(s)]
        self.cnt = cnt
        self.hpos = torch.nonzero(hard.reshape(-1)).reshape(-1)


class _Exact:
    """The step in 64 bits, with the step size and the constants rounded to 32 bits as the library's interface gives
    them.  The fields hold 0 at walls, so a wall neighbour's mirror value is the centre times their number."""

    def __init__(self, c, i, grid=None):
        dev = _device()
        f = np.float32
        self.g = g = grid or _Grid(c, dev)
        self.c, self.dev = c, dev
        dt = f(f(_courant(c)) * f(H)) / f(f(C0) * np.sqrt(f(3)))
        self.lam2 = float(f(f(f(f(C0) * f(C0)) * dt) * dt)) * float(f(1) / f(f(H) * f(H)))
        self.K = float(f(f(f(f(C0) * dt) / f(H)) * f(0.95)))
        self.kgw = self.K * float(f(0.4)) * g.weight
        self.coef = torch.tensor(i["coef"].astype(np.float64), device=dev)
        self.src = torch.tensor(_index(c, i["src"]).astype(np.int64), device=dev)
        self.rcv = torch.tensor(_index(c, i["rcv"]).astype(np.int64), device=dev)
        self.sig = torch.tensor(i["sig"].astype(np.float64), device=dev)
        self.hard = i["hard"]
        self.p = torch.zeros(g.shape, dtype=torch.float64, device=dev)
        self.q = torch.zeros_like(self.p)
        if i["sphere"]:
            x, y, z, r, v = i["sphere"]
            ax = [torch.arange(e, device=dev, dtype=torch.int64) for e in g.shape]
            d2 = (ax[0] - z)[:, None, None] ** 2 + (ax[1] - y)[None, :, None] ** 2 + (ax[2] - x)[None, None, :] ** 2
            self.p[d2 <= r * r] = float(f(v))
        self.x = [torch.zeros((2, len(g.bnd)), dtype=torch.float64, device=dev) for _ in range(c["sections"] + 1)]

    def filtered(self, x, d, coef):
        """(output, new states) of the cascades on d; x holds the last two values of every section's input and of
        the last output."""
        new, v = [], d
        for s in range(self.c["sections"]):
            k = coef[self.g.mat, s]
            y = k[:, 0] * v + k[:, 1] * x[s][0] + k[:, 2] * x[s][1] - k[:, 3] * x[s + 1][0] - k[:, 4] * x[s + 1][1]
            new.append(torch.stack([v, x[s][0]]))
            v = y
        new.append(torch.stack([v, x[-1][0]]))
        return v, new

    def corrected(self, r, p, q, y):
        if self.c["kind"] == "calls":
            return r - self.kgw * (0.1 * y + 0.9 * (p - q))
        a = 0.45 * self.kgw
        return (r - self.kgw * 0.1 * y + a * q) / (1 + a)

    def free(self, p, q):
        """p+ of the inner voxels before the filters."""
        s = p[1:-1, 1:-1, 2:] + p[1:-1, 1:-1, :-2]
        s = s + p[1:-1, 2:, 1:-1]
        s = s + p[1:-1, :-2, 1:-1]
        s = s + p[2:, 1:-1, 1:-1]
        s = s + p[:-2, 1:-1, 1:-1]
        m = p[1:-1, 1:-1, 1:-1]
        s = s + (self.g.cnt - 6.0) * m
        s = s * self.lam2 + 2 * m
        s = s - q[1:-1, 1:-1, 1:-1]
        return s.masked_fill(self.g.keep, 0.0)

    def step(self, n):
        """One step in place; the receiver samples."""
        g, p, q = self.g, self.p, self.q
        pb, qb = p.reshape(-1)[g.bnd], q.reshape(-1)[g.bnd]
        r = self.free(p, q)
        q[1:-1, 1:-1, 1:-1] = r
        del r
        new = q.reshape(-1)
        y, self.x = self.filtered(self.x, pb - qb, self.coef)
        new[g.bnd] = self.corrected(new[g.bnd], pb, qb, y)
        if len(g.hpos):
            new[g.hpos] = float(self.hard[n]) if n < len(self.hard) else 0.0
        if len(self.src) and n < self.sig.shape[1]:
            new[self.src] += self.sig[:, n]
        self.p, self.q = q, p
        return new[self.rcv]

    def run(self, steps):
        return torch.stack([self.step(n) for n in range(steps)], 1)


def _exact_gradient(c, i):
    from torch.utils.checkpoint import checkpoint

    e = _Exact(c, i)
    g = e.g
    coef = e.coef.clone().requires_grad_(True)
    sig = e.sig.clone().requires_grad_(True)
    inner = torch.zeros(g.shape, dtype=torch.bool, device=e.dev)
    inner[1:-1, 1:-1, 1:-1] = True

    def steps(p, q, coef, sig, n0, n1, *x):
        x, out = list(x), []
        for n in range(n0, n1):
            pb, qb = p.reshape(-1)[g.bnd], q.reshape(-1)[g.bnd]
            r = torch.nn.functional.pad(e.free(p, q), (1,) * 6).reshape(-1)
            y, x = e.filtered(x, pb - qb, coef)
            r = r.index_put((g.bnd,), e.corrected(r[g.bnd], pb, qb, y))
            r = r.index_put((e.src,), sig[:, n], accumulate=True)
            out.append(r[e.rcv])
            p, q = r.reshape(g.shape), p
        return (p, q, torch.stack(out, 1), *x)

    p, q, x, irs = e.p, e.q, e.x, []
    for n0 in range(0, c["steps"], 8):
        p, q, ir, *x = checkpoint(steps, p, q, coef, sig, n0, min(n0 + 8, c["steps"]), *x, use_reentrant=False)
        irs.append(ir)
    ir = torch.cat(irs, 1)
    gc, gs = torch.autograd.grad((ir * torch.tensor(i["loss"], dtype=torch.float64, device=e.dev)).sum(), (coef, sig))
    return dict(ir=ir.detach().cpu(), coef=gc.cpu(), signal=gs.cpu())


def _exact_resampled(c, seed):
    t, i = _trace_inputs(c, seed)
    x = _Exact(t, i).run(c["steps"]).cpu().numpy()
    f = np.float32
    dt = float(f(f(_courant(t)) * f(H)) / f(f(C0) * np.sqrt(f(3))))
    length = int(c["rate"] * (c["steps"] * dt))
    y = x
    for b0, b1, b2, _, a1, a2 in _sos(c):
        z1 = z2 = np.zeros(len(y))
        o = np.zeros_like(y)
        for n in range(y.shape[1]):
            v = y[:, n]
            o[:, n] = b0 * v + z1
            z1 = b1 * v - a1 * o[:, n] + z2
            z2 = b2 * v - a2 * o[:, n]
        y = o
    at = np.arange(length) / c["rate"] / dt
    lo = np.minimum(at.astype(np.int64), c["steps"] - 1)
    hi = np.minimum(lo + 1, c["steps"] - 1)
    linear = y[:, lo] * (1 - (at - lo)) + y[:, hi] * (at - lo)
    dev = _device()
    half, beta, cutoff = c["half"], 10.06, 0.9167
    xt = torch.tensor(x, device=dev)
    fc2 = cutoff * min(1.0, c["rate"] * dt)
    out = []
    for k in range(0, length, 1024):
        pos = torch.arange(k, min(length, k + 1024), device=dev, dtype=torch.float64) / c["rate"] / dt
        n = torch.floor(pos)[:, None] + torch.arange(-half, half + 2, device=dev)
        tau = pos[:, None] - n
        u = tau / half
        ok = (n >= 0) & (n < c["steps"]) & (u.abs() < 1)
        w = torch.special.i0(beta * torch.sqrt((1 - u * u).clamp(min=0))) / torch.special.i0(
            torch.tensor(beta, device=dev, dtype=torch.float64))
        tap = torch.where(ok, fc2 * torch.sinc(fc2 * tau) * w, 0.0)
        v = xt[:, n.clamp(0, c["steps"] - 1).to(torch.int64)]
        out.append((v * tap).sum(-1))
    sinc = torch.cat(out, 1).cpu().numpy()

    def normal(a):
        peak = np.abs(a).max(1, keepdims=True)
        return a / np.where(peak > 0, peak, 1.0)

    return [normal(linear), normal(sinc)]


def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "setup":
        return None  # whole numbers, and weights that are a function of them
    if k == "resample":
        return _exact_resampled(c, seed)
    if k == "batch":
        return [_Exact(m, _inputs(m, seed * 1000 + j)).run(c["steps"]).cpu() for j, m in enumerate(_members(c))]
    i = _inputs(c, seed)
    if k == "gradient":
        return _exact_gradient(c, i)
    out = _Exact(c, i).run(c["steps"]).cpu()
    return out[0] if k == "calls" else out
