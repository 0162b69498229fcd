"""Performance cases of the step library: what programs that link it have it do.

Four kinds of work, each through the public entry points:

  world     b2World_Step of one world followed by b2World_GetBodyStates, as a game or a
            robotics loop does once a frame (a scene name and its sizes)
  batch     a rollout of b2World_StepBatch over many independent worlds, then every
            world's body states (parameter sweeps, reinforcement-learning environments)
  gradient  b2World_StepBackwardBatch over recorded worlds (the backward pass of the
            drop-boxes harness in box2c_gb300/autograd.py)
  solve     b2SolveContacts / b2SolveContactsNoAlloc on device buffers, for engines that
            do their own collision detection: each pass copies new inputs into the
            buffers and solves them

Sizes are those of the repository's benchmark and parity scenes and of the ranges around
them.
"""
import ctypes as C
import math

import numpy as np
import torch

import box2c_gb300
from box2c_gb300 import autograd
from box2c_gb300.capi import (MANIFOLD_BYTES, BodyId, ContactSolveDesc, Vec2, bind_batch_api, bind_gpu_api, bind_solve_api,
                              world_array)

DT = 1.0 / 60.0
SUBSTEPS = 4
COLORS = 12
OVERFLOW = 11
NO_ALLOC_MAX = 16384


def listed():
    return [
        # a small stack in a game level: latency and launches count
        {"name": "world_pyramid_20", "kind": "world", "scene": "pyramid", "size": 20},
        # the benchmark's large pyramid, one big island
        {"name": "world_pyramid_100", "kind": "world", "scene": "pyramid", "size": 100},
        # the reference benchmark's many pyramids: 22000 bodies, too many for one cluster
        {"name": "world_many_pyramids_20", "kind": "world", "scene": "many_pyramids", "size": 20},
        # the benchmark's tumbler: boxes and circles, a motor, contacts that change every
        # step, and a body with more contacts than there are graph colours
        {"name": "world_tumbler_2000", "kind": "world", "scene": "tumbler", "size": 2000},
        # the reference benchmark's joint grid, hanging: 9900 circles and 19800 joints
        {"name": "world_joint_grid_100", "kind": "world", "scene": "joint_grid", "size": 100},
        # capsules, circles, boxes and rounded boxes piled in a funnel of segments
        {"name": "world_shape_pile_600", "kind": "world", "scene": "shape_pile", "size": 600},
        # the batched benchmark's uneven pyramids (bases 4 to 40), ten steps a read
        {"name": "batch_pyramids_160", "kind": "batch", "scene": "pyramids", "worlds": 160, "low": 4, "high": 40, "steps": 10},
        # small learning environments: eight mixed bodies each, thirty steps a read
        {"name": "batch_drop_96", "kind": "batch", "scene": "drop", "worlds": 96, "low": 8, "high": 8, "steps": 30},
        # the differentiable benchmark's backward pass: eight boxes, 120 recorded steps
        {"name": "gradient_96", "kind": "gradient", "worlds": 96, "boxes": 8, "steps": 120},
        # an engine's small contact set, in the form that allocates nothing
        {"name": "solve_900", "kind": "solve", "contacts": 900, "lid": 0, "alloc": False},
        # a set near the large pyramid's, with a lid that overflows the colours
        {"name": "solve_15000", "kind": "solve", "contacts": 15000, "lid": 24, "alloc": True},
        # a large set
        {"name": "solve_60000", "kind": "solve", "contacts": 60000, "lid": 0, "alloc": True},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["world", "world", "world", "batch", "gradient", "solve", "solve"])
    if kind == "world":
        scene = rng.choice(["pyramid", "pyramid", "many_pyramids", "tumbler", "joint_grid", "shape_pile"])
        low, high = {"pyramid": (5, 150), "many_pyramids": (3, 20), "tumbler": (50, 2000), "joint_grid": (10, 100),
                     "shape_pile": (30, 600)}[scene]
        return {"kind": kind, "scene": scene, "size": _log_int(rng, low, high)}
    if kind == "batch":
        if rng.random() < 0.5:
            low = rng.randint(4, 12)
            return {"kind": kind, "scene": "pyramids", "worlds": _log_int(rng, 16, 140), "low": low, "high": rng.randint(low, 40),
                    "steps": rng.randint(4, 10)}
        boxes = rng.randint(3, 12)
        return {"kind": kind, "scene": "drop", "worlds": _log_int(rng, 16, 96), "low": boxes, "high": boxes, "steps": rng.randint(10, 30)}
    if kind == "gradient":
        return {"kind": kind, "worlds": _log_int(rng, 8, 96), "boxes": rng.randint(3, 8), "steps": rng.randint(20, 120)}
    contacts = _log_int(rng, 60, 60000)
    return {"kind": kind, "contacts": contacts, "lid": rng.choice([0, 0, 9, 17, 24]) if contacts > 1000 else 0,
            "alloc": contacts > 12000 or rng.random() < 0.6}


# ---------------------------------------------------------------------------- worlds
class Worlds:
    """Worlds that live as long as the state that holds them."""

    def __init__(self, backend, ids):
        self.backend = backend
        self.ids = ids

    def __del__(self):
        for w in self.ids:
            self.backend.destroy(w)


def _backend():
    g = box2c_gb300.load()
    bind_gpu_api(g.lib)
    bind_batch_api(g.lib)
    bind_solve_api(g.lib)
    g.lib.b2SolveContactsNoAlloc.argtypes = [C.POINTER(ContactSolveDesc)]
    g.lib.b2SolveContactsNoAlloc.restype = C.c_int
    return g


def _body_count(g, world):
    return g.lib.b2World_GetBodyStates(world, None, 0)


def _nudge(g, world, rng, count):
    """Small velocities on some of the world's bodies (ids are given in creation order)."""
    n = _body_count(g, world)
    for i in sorted(set(int(b) for b in rng.integers(0, n, count))):
        body = BodyId(i + 1, world.index1 - 1, 1)
        if g.lib.b2Body_IsValid(body):
            g.lib.b2Body_SetLinearVelocity(body, Vec2(float(rng.uniform(-0.2, 0.2)), float(rng.uniform(0.0, 0.2))))


def _make_world(g, case, seed):
    scene, size = case["scene"], case["size"]
    rng = np.random.default_rng(seed)
    if scene == "pyramid":
        return g.pyramid(size, 0.01, seed)
    if scene == "many_pyramids":
        w = g.many_pyramids(size, size, 10)
        _nudge(g, w, rng, 64)
        return w
    if scene == "tumbler":
        return g.tumbler(size, seed, 0)
    if scene == "joint_grid":
        return g.joint_grid(size, -float(rng.uniform(9.0, 11.0)))
    return g.shape_pile(size, seed)


def _batch_sizes(case):
    """Pyramid bases (or body counts) of the batch's worlds; the case's, not the seed's."""
    rng = np.random.default_rng(case["worlds"] * 1000003 + case["low"] * 101 + case["high"])
    return [int(x) for x in rng.integers(case["low"], case["high"] + 1, case["worlds"])]


def _prepare_world(case, seed):
    g = _backend()
    held = Worlds(g, [_make_world(g, case, seed)])
    world = held.ids[0]
    g.step(world, DT, SUBSTEPS, 3)
    out = np.zeros((_body_count(g, world), 7), np.float32)
    return {"kind": "world", "lib": g.lib, "held": held, "world": world, "out": out, "ptr": out.ctypes.data, "n": len(out)}


def _run_world(s):
    lib = s["lib"]
    lib.b2World_Step(s["world"], DT, SUBSTEPS)
    lib.b2World_GetBodyStates(s["world"], s["ptr"], s["n"])
    return s["out"]


def _prepare_batch(case, seed):
    g = _backend()
    rng = np.random.default_rng(seed)
    worlds = []
    for i, n in enumerate(_batch_sizes(case)):
        if case["scene"] == "pyramids":
            worlds.append(g.pyramid(n, 0.005, seed + i))
        else:
            worlds.append(g.drop_boxes(rng.uniform(1, 5, n), rng.normal(0, 1, n), rng.normal(0, 1, n), float(rng.uniform(0.2, 0.9)),
                                       np.arange(n) % 3))
    held = Worlds(g, worlds)
    counts = [_body_count(g, w) for w in worlds]
    out = np.zeros((sum(counts), 7), np.float32)
    at = np.concatenate([[0], np.cumsum(counts)[:-1]])
    reads = [(w, out.ctypes.data + 28 * int(a), n) for w, a, n in zip(worlds, at, counts)]
    ids = world_array(worlds)
    g.lib.b2World_StepBatch(ids, len(worlds), DT, SUBSTEPS)
    return {"kind": "batch", "lib": g.lib, "held": held, "ids": ids, "n": len(worlds), "steps": case["steps"], "reads": reads, "out": out}


def _run_batch(s):
    lib = s["lib"]
    for _ in range(s["steps"]):
        lib.b2World_StepBatch(s["ids"], s["n"], DT, SUBSTEPS)
    for world, ptr, n in s["reads"]:
        lib.b2World_GetBodyStates(world, ptr, n)
    return s["out"]


class Drop(autograd.DropBoxes):
    """The drop-boxes harness, whose worlds go when the state does."""

    def __del__(self):
        self.destroy()


def _prepare_gradient(case, seed):
    g = _backend()
    rng = np.random.default_rng(seed)
    n, boxes = case["worlds"], case["boxes"]
    sim = Drop(g, rng.uniform(1, 5, (n, boxes)), steps=case["steps"], substeps=SUBSTEPS, dt=DT)
    v0 = rng.normal(0, 1, (n, boxes, 2)).astype(np.float32)
    mu = rng.uniform(0.2, 0.9, n).astype(np.float32)
    p = sim.run(v0, mu, record=True)
    return {"kind": "gradient", "sim": sim, "grad": 2.0 * p}


def _run_gradient(s):
    gv, gmu = s["sim"].backward(s["grad"])
    return {"velocity": gv, "friction": gmu}


# ---------------------------------------------------------------------------- solve
POINT = np.dtype([("point", "f4", 2), ("anchorA", "f4", 2), ("anchorB", "f4", 2), ("separation", "f4"), ("normalImpulse", "f4"),
                  ("tangentImpulse", "f4"), ("maxNormalImpulse", "f4"), ("normalVelocity", "f4"), ("id", "u2"), ("persisted", "u1"),
                  ("pad", "u1")])
MANIFOLD = np.dtype([("pts", POINT, 2), ("normal", "f4", 2), ("count", "i4")])
assert MANIFOLD.itemsize == MANIFOLD_BYTES


def _wall(case):
    """A brick wall of unit boxes on a static floor, coloured so that no two contacts of a
    colour share a box: each box rests on two of the course below and leans on its
    neighbours; an optional heavy lid lies on `lid` boxes of the top course, and those of
    its contacts that find no free colour overflow.  About `contacts` contacts; which
    joints of the wall are open is the case's, not the seed's.  Returns (boxes, lid id or
    -1, contacts) with one row (a, b, kind, colour, course) per contact, in solve order."""
    rng = np.random.default_rng(case["contacts"] * 31 + case["lid"])
    boxes = max(6, int(case["contacts"] / 2.62))
    width = max(3, int(math.sqrt(boxes * 2)), case["lid"] + 1)
    height = max(2, boxes // width)
    boxes = width * height
    rows = [(-1, c, 0, 6, 0) for c in range(width)]
    r, c = np.divmod(np.arange(boxes - width), width)
    low = r * width + c
    straight = np.stack([low, low + width, np.full_like(low, 1), r % 2, r], 1)
    side = np.where(r % 2 == 0, c - 1, c + 1)
    ok = (side >= 0) & (side < width)
    diagonal = np.stack([low, (r + 1) * width + side, np.where(r % 2 == 0, 2, 3), 2 + r % 2, r], 1)[ok]
    r, c = np.divmod(np.arange(boxes), width)
    at = r * width + c
    lean = np.stack([at, at + 1, np.full_like(at, 4), 4 + c % 2, r], 1)[c < width - 1]
    lean = lean[rng.random(len(lean)) < 0.7]
    table = np.concatenate([np.array(rows), straight, diagonal, lean])
    lid = -1
    if case["lid"]:
        lid = boxes
        top = (height - 1) * width
        below = (height - 2) % 2
        free = [x for x in (1 - below, 3 - below, 6, 7, 8, 9, 10)]
        pairs = [(top + k, lid, 5, free[k] if k < len(free) else OVERFLOW, height) for k in range(case["lid"])]
        table = np.concatenate([table, np.array(pairs)])
    return boxes, lid, table[np.argsort(table[:, 3], kind="stable")]


def _solve_inputs(case, seed):
    boxes, lid, table = _wall(case)
    rng = np.random.default_rng(seed)
    n, nb = len(table), boxes + (lid >= 0)
    kind, course = table[:, 2], table[:, 4]
    states = np.zeros((nb, 8), np.float32)
    states[:, 0:2] = rng.normal(0, 0.05, (nb, 2))
    states[:, 2] = rng.normal(0, 0.05, nb)
    states[:, 6] = 1.0
    mass = np.tile(np.array([1.0, 1.0, 1.0 / 6.0, 6.0], np.float32), (nb, 1))
    forces = np.zeros((nb, 4), np.float32)
    forces[:, 0] = rng.normal(0, 0.1, nb)
    forces[:, 3] = 1.0
    damping = np.zeros((nb, 4), np.float32)
    damping[:, 0:2] = rng.choice([0.0, 0.05], (nb, 2))
    if lid >= 0:
        mass[lid] = (20.0, 1.0 / 20.0, 800.0, 1.0 / 800.0)
    m = np.zeros(n, MANIFOLD)
    tilt = rng.normal(0, 0.01, n)
    upright = kind != 4
    m["normal"][:, 0] = np.where(upright, np.sin(tilt), np.cos(tilt))
    m["normal"][:, 1] = np.where(upright, np.cos(tilt), np.sin(tilt))
    m["count"] = np.where(rng.random(n) < 0.9, 2, 1)
    # offset of B's centre from A's, and the two ends of their common face
    dx = np.select([kind == 2, kind == 3, kind == 4], [-0.5, 0.5, 1.0], 0.0)
    lo = np.where(upright, np.maximum(-0.5, dx - 0.5), -0.5)
    hi = np.where(upright, np.minimum(0.5, dx + 0.5), 0.5)
    load = np.where(upright, 0.17 * (course.max() + 1 - course) / 4.0, 0.01)
    first = int(table[kind == 5, 0].min()) if lid >= 0 else 0
    lid_x = np.where(kind == 5, table[:, 0] - first - 0.5 * case["lid"] + 0.5, 0.0)
    for j in (0, 1):
        p = m["pts"][:, j]
        along = (hi if j else lo) + rng.normal(0, 0.003, n)
        p["anchorA"][:, 0] = np.where(upright, along, 0.5)
        p["anchorA"][:, 1] = np.where(upright, 0.5, along)
        p["anchorB"][:, 0] = np.where(upright, along - dx + lid_x, -0.5)
        p["anchorB"][:, 1] = np.where(upright, -0.5, along)
        p["separation"] = rng.normal(-0.003, 0.003, n)
        p["normalImpulse"] = load * rng.uniform(0.5, 1.5, n)
        p["tangentImpulse"] = 0.1 * p["normalImpulse"] * rng.uniform(-1, 1, n)
        p["id"] = j + 1
        p["persisted"] = 1
        for f in ("anchorA", "anchorB", "separation", "normalImpulse", "tangentImpulse", "id", "persisted"):
            p[f][m["count"] <= j] = 0
    mix = np.zeros((n, 2), np.float32)
    mix[:, 0] = rng.uniform(0.2, 0.9, n)
    mix[:, 1] = np.where(rng.random(n) < 0.2, 0.3, 0.0)
    start = np.searchsorted(table[:, 3], np.arange(COLORS + 1))
    return {"states": states, "mass": mass, "forces": forces, "damping": damping, "awake": np.arange(nb, dtype=np.int32),
            "pairs": np.ascontiguousarray(table[:, :2], np.int32), "mix": mix, "manifolds": m, "start": [int(x) for x in start]}


def _prepare_solve(case, seed):
    g = _backend()
    a = _solve_inputs(case, seed)
    n = len(a["pairs"])
    t = {k: torch.from_numpy(a[k]).cuda() for k in ("states", "mass", "forces", "damping", "awake", "pairs", "mix")}
    t["manifolds"] = torch.from_numpy(a["manifolds"].view(np.float32).reshape(n, MANIFOLD_BYTES // 4)).cuda()
    states, manifolds = t["states"].clone(), t["manifolds"].clone()
    d = ContactSolveDesc()
    d.states, d.manifolds = states.data_ptr(), manifolds.data_ptr()
    d.massData, d.forces, d.damping = t["mass"].data_ptr(), t["forces"].data_ptr(), t["damping"].data_ptr()
    d.bodies, d.bodyCount = t["awake"].data_ptr(), len(a["awake"])
    d.contactBodies, d.contactMix, d.contactCount = t["pairs"].data_ptr(), t["mix"].data_ptr(), n
    for c in range(COLORS + 1):
        d.colorStart[c] = a["start"][c]
    d.timeStep, d.subStepCount, d.gravity = DT, SUBSTEPS, Vec2(0.0, -10.0)
    d.contactHertz, d.contactDampingRatio, d.contactPushout, d.restitutionThreshold = 30.0, 10.0, 3.0, 1.0
    d.enableWarmStarting = True
    d.stream = None
    fn = g.lib.b2SolveContacts if case["alloc"] or n > NO_ALLOC_MAX else g.lib.b2SolveContactsNoAlloc
    return {"kind": "solve", "fn": fn, "desc": d, "arg": C.byref(d), "inputs": t, "states": states, "manifolds": manifolds}


def _run_solve(s):
    s["states"].copy_(s["inputs"]["states"])
    s["manifolds"].copy_(s["inputs"]["manifolds"])
    rc = s["fn"](s["arg"])
    if rc != 0:
        raise RuntimeError(f"contact solve failed: {rc}")
    return {"states": s["states"], "manifolds": s["manifolds"]}


def prepare(case, seed):
    return {"world": _prepare_world, "batch": _prepare_batch, "gradient": _prepare_gradient, "solve": _prepare_solve}[case["kind"]](case, seed)


def run(state):
    return {"world": _run_world, "batch": _run_batch, "gradient": _run_gradient, "solve": _run_solve}[state["kind"]](state)


# ---------------------------------------------------------------------------- work
# bytes a step must move once: a body's state, pose, mass, force, extents, boxes and shape
# (read, and the written part of them), its read-back; a contact's shapes, mixed material
# and manifold read and written; a joint's record read and written
BODY_BYTES, CONTACT_BYTES, JOINT_BYTES = 560, 260, 512
# operations of a step: manifold, preparation, four substeps and restitution of a contact;
# integration and finalisation of a body; four substeps of a joint
BODY_FLOPS, CONTACT_FLOPS, JOINT_FLOPS = 300, 2600, 1600
SOLVE_BODY_BYTES, SOLVE_CONTACT_BYTES = 116, 164
SOLVE_BODY_FLOPS, SOLVE_CONTACT_FLOPS = 120, 2200


def _pyramid_contacts(base):
    return base + 3 * base * (base - 1) // 2


def _counts(case):
    """Bodies, contacts and joints of one step of the case."""
    if case["kind"] == "world":
        scene, n = case["scene"], case["size"]
        if scene == "pyramid":
            return n * (n + 1) // 2, _pyramid_contacts(n), 0
        if scene == "many_pyramids":
            return 55 * n * n, _pyramid_contacts(10) * n * n, 0
        if scene == "joint_grid":
            return n * n, 0, 2 * n * (n - 1)
        return n, int(2.2 * n), int(scene == "tumbler")
    sizes = _batch_sizes(case)
    if case["scene"] == "pyramids":
        return sum(n * (n + 1) // 2 for n in sizes), sum(_pyramid_contacts(n) for n in sizes), 0
    return sum(sizes), sum(2 * n for n in sizes), 0


def work(case):
    if case["kind"] == "solve":
        boxes, lid, table = _wall(case)
        nb = boxes + (lid >= 0)
        return {"bytes": nb * SOLVE_BODY_BYTES + len(table) * SOLVE_CONTACT_BYTES,
                "flops": nb * SOLVE_BODY_FLOPS + len(table) * SOLVE_CONTACT_FLOPS}
    if case["kind"] == "gradient":
        steps = case["worlds"] * case["steps"]
        # the tape read once (64 bytes a body, 144 a row), the gradients written; replay
        # and reverse of every row
        return {"bytes": steps * case["boxes"] * (64 + 1.5 * 144) + case["worlds"] * case["boxes"] * 48,
                "flops": steps * case["boxes"] * (1.5 * 4 * CONTACT_FLOPS + 4 * BODY_FLOPS)}
    steps = case.get("steps", 1)
    b, c, j = _counts(case)
    return {"bytes": steps * (b * BODY_BYTES + c * CONTACT_BYTES + j * JOINT_BYTES),
            "flops": steps * (b * BODY_FLOPS + c * CONTACT_FLOPS + j * JOINT_FLOPS)}


# ---------------------------------------------------------------------------- exact
def exact(case, seed):
    """The contact solve in 64 bits (soft steps, one colour at a time, the overflow set
    first and one contact after another).  Whole worlds have no such value: their contacts
    come and go, and a step after the first differs with the rounding of the one before."""
    if case["kind"] != "solve":
        return None
    a = _solve_inputs(case, seed)
    f = np.float64
    dt, sub = f(np.float32(DT)), SUBSTEPS
    h, inv_h = dt / sub, sub / dt
    st = a["states"].astype(f)
    m, pairs, start = a["manifolds"], a["pairs"], a["start"]
    n = len(pairs)
    mass = np.concatenate([a["mass"].astype(f), np.zeros((1, 4))])  # index -1: the static body
    st = np.concatenate([st, [[0, 0, 0, 0, 0, 0, 1, 0]]]).astype(f)

    def soft(hertz, zeta):
        omega = 2 * math.pi * hertz
        a1 = 2 * zeta + h * omega
        a2 = h * omega * a1
        return omega / a1, a2 / (1 + a2), 1 / (1 + a2)

    hertz = min(30.0, 0.25 * inv_h)
    on_static = (pairs < 0).any(1)
    rate, mscale, iscale = (np.where(on_static, s, c) for s, c in zip(soft(2 * hertz, 10.0), soft(hertz, 10.0)))
    ia, ib = pairs[:, 0], pairs[:, 1]
    mA, iA, mB, iB = mass[ia, 1], mass[ia, 3], mass[ib, 1], mass[ib, 3]
    nx, ny = m["normal"][:, 0].astype(f), m["normal"][:, 1].astype(f)
    tx, ty = ny, -nx
    fric, rest = a["mix"][:, 0].astype(f), a["mix"][:, 1].astype(f)
    P = []
    for j in (0, 1):
        p = m["pts"][:, j]
        on = m["count"] > j
        ax, ay, bx, by = (p[k][:, i].astype(f) * on for k in ("anchorA", "anchorB") for i in (0, 1))
        rn_a, rn_b, rt_a, rt_b = ax * ny - ay * nx, bx * ny - by * nx, ax * ty - ay * tx, bx * ty - by * tx
        kn, kt = mA + mB + iA * rn_a ** 2 + iB * rn_b ** 2, mA + mB + iA * rt_a ** 2 + iB * rt_b ** 2
        dvx = (st[ib, 0] - st[ib, 2] * by) - (st[ia, 0] - st[ia, 2] * ay)
        dvy = (st[ib, 1] + st[ib, 2] * bx) - (st[ia, 1] + st[ia, 2] * ax)
        P.append({"on": on, "ax": ax, "ay": ay, "bx": bx, "by": by, "base": on * (p["separation"] - ((bx - ax) * nx + (by - ay) * ny)),
                  "nm": on / kn, "tm": on / kt, "rv": on * (dvx * nx + dvy * ny), "ni": p["normalImpulse"].astype(f) * on,
                  "ti": p["tangentImpulse"].astype(f) * on, "mx": np.zeros(n)})

    def push(k, p, px, py):
        A, B = ia[k], ib[k]
        st[A, 0] -= mA[k] * px
        st[A, 1] -= mA[k] * py
        st[A, 2] -= iA[k] * (p["ax"][k] * py - p["ay"][k] * px)
        st[B, 0] += mB[k] * px
        st[B, 1] += mB[k] * py
        st[B, 2] += iB[k] * (p["bx"][k] * py - p["by"][k] * px)

    def relative(k, p):
        A, B = ia[k], ib[k]
        return ((st[B, 0] - st[B, 2] * p["by"][k]) - (st[A, 0] - st[A, 2] * p["ay"][k]),
                (st[B, 1] + st[B, 2] * p["bx"][k]) - (st[A, 1] + st[A, 2] * p["ax"][k]))

    def stage(k, phase, serial):
        """phase: 0 warm start, 1 solve, 2 relax, 3 restitution, of contacts k."""
        if phase == 3 and serial and rest[k][0] == 0:
            return
        A, B = ia[k], ib[k]
        for p in P:
            if phase == 0:
                push(k, p, p["ni"][k] * nx[k] + p["ti"][k] * tx[k], p["ni"][k] * ny[k] + p["ti"][k] * ty[k])
                continue
            dvx, dvy = relative(k, p)
            vn = dvx * nx[k] + dvy * ny[k]
            if phase == 3:
                skip = (p["rv"][k] + 1.0 > 0) | (p["mx"][k] == 0)
                new = np.maximum(p["ni"][k] - np.where(skip, 0, p["nm"][k]) * (vn + rest[k] * p["rv"][k]), 0)
            else:
                rax, ray = st[A, 6] * p["ax"][k] - st[A, 7] * p["ay"][k], st[A, 7] * p["ax"][k] + st[A, 6] * p["ay"][k]
                rbx, rby = st[B, 6] * p["bx"][k] - st[B, 7] * p["by"][k], st[B, 7] * p["bx"][k] + st[B, 6] * p["by"][k]
                sx, sy = st[B, 4] - st[A, 4] + rbx - rax, st[B, 5] - st[A, 5] + rby - ray
                s = sx * nx[k] + sy * ny[k] + p["base"][k]
                use = phase == 1
                ms, im = (mscale[k], iscale[k]) if use else (np.ones(len(k)), np.zeros(len(k)))
                if serial:
                    ms, im = np.where(s > 0, 1, ms), np.where(s > 0, 0, im)
                bias = np.where(s > 0, s * inv_h, np.maximum(rate[k] * s, -3.0) if use else 0)
                new = np.maximum(p["ni"][k] - (p["nm"][k] * ms * (vn + bias) + im * p["ni"][k]), 0)
            impulse = np.where(p["on"][k], new - p["ni"][k], 0)
            p["ni"][k] += impulse
            if phase != 3 or serial:
                p["mx"][k] = np.maximum(p["mx"][k], impulse if serial else p["ni"][k])
            push(k, p, impulse * nx[k], impulse * ny[k])
        if phase in (1, 2):
            for p in P:
                dvx, dvy = relative(k, p)
                top = fric[k] * p["ni"][k]
                new = np.clip(p["ti"][k] - p["tm"][k] * (dvx * tx[k] + dvy * ty[k]), -top, top)
                impulse = np.where(p["on"][k], new - p["ti"][k], 0)
                p["ti"][k] += impulse
                push(k, p, impulse * tx[k], impulse * ty[k])
        st[-1] = (0, 0, 0, 0, 0, 0, 1, 0)

    def sweep(phase):
        for k in range(start[OVERFLOW], n):
            stage(np.array([k]), phase, True)
        for c in range(OVERFLOW):
            if start[c + 1] > start[c]:
                stage(np.arange(start[c], start[c + 1]), phase, False)

    b = a["awake"]
    fo, da, ms = a["forces"].astype(f), a["damping"].astype(f), mass
    for _ in range(sub):
        ld, ad = 1 / (1 + h * da[b, 0]), 1 / (1 + h * da[b, 1])
        st[b, 0] = (h * ms[b, 1] * fo[b, 0]) + ld * st[b, 0]
        st[b, 1] = (h * ms[b, 1] * (fo[b, 1] + ms[b, 0] * fo[b, 3] * -10.0)) + ld * st[b, 1]
        st[b, 2] = h * ms[b, 3] * fo[b, 2] + ad * st[b, 2]
        sweep(0)
        sweep(1)
        c, s = st[b, 6] - h * st[b, 2] * st[b, 7], st[b, 7] + h * st[b, 2] * st[b, 6]
        mag = np.hypot(c, s)
        st[b, 6], st[b, 7] = c / mag, s / mag
        st[b, 4:6] += h * st[b, 0:2]
        sweep(2)
    sweep(3)
    out = m.view(np.float32).reshape(n, MANIFOLD_BYTES // 4).astype(f)
    for j, p in enumerate(P):
        # contacts in the colours store both points, the others their own
        put = (np.arange(n) < start[OVERFLOW]) | p["on"]
        for o, key in ((7, "ni"), (8, "ti"), (9, "mx"), (10, "rv")):
            out[put, 12 * j + o] = p[key][put]
    return {"states": st[:-1], "manifolds": out}
