"""The resident contact solver (csrc/resident.cu) at the edges of its spaces: one CTA, a
cluster, a cooperative grid, body indices that do not fit on chip, overflow rows and an
empty set.  The reference is the oracle's captured solver stage; tolerance: none."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from box2c_gb300.capi import bind_solve_api
from tests.helpers import lockstep
from tests.test_gpu_solve_api import capture_step, make_desc, solve_on_device


def _scene(oracle, name):
    if name == "plank":  # a plank under sixteen boxes: contacts beyond the graph colours
        n = 17
        heights = np.array([0.2] + [0.9 + 0.01 * (k % 3) for k in range(n - 1)], np.float32)
        kinds = np.array([3] + [0] * (n - 1), np.int32)
        return oracle.drop_boxes(heights, np.zeros(n), np.zeros(n), 0.6, kinds), 30
    if name == "many":
        return oracle.many_pyramids(20, 20, 10), 3
    size = int(name)
    return oracle.pyramid(size, 0.01, 5), 12


def _spread(cap, stride):
    """The same set with body indices spread over `stride` times as many states."""
    n = len(cap["statesIn"])
    out = dict(cap)
    for k in ("statesIn", "statesOut", "mass", "force", "damping"):
        a = np.zeros((n * stride, cap[k].shape[1]), np.float32)
        a[::stride] = cap[k]
        out[k] = a
    out["awake"] = cap["awake"] * stride
    out["contactBodies"] = np.where(cap["contactBodies"] < 0, -1, cap["contactBodies"] * stride).astype(np.int32)
    return out


# one CTA up to about 1300 contacts, a cluster up to about 22000, a grid above; 30 and 21
# lie on both sides of the first line, 120 above the second; strides 40 and 90 put the
# indices beyond the cluster's body slots and beyond 2^16
@pytest.mark.gpu
@pytest.mark.parametrize("scene,stride", [("1", 1), ("21", 1), ("30", 1), ("100", 1), ("120", 1), ("many", 1), ("plank", 1),
                                          ("plank", 700), ("21", 90), ("40", 40), ("40", 90)])
def test_resident_solver_matches_oracle(gpu, oracle, scene, stride):
    torch = pytest.importorskip("torch")
    w, warm = _scene(oracle, scene)
    oracle.step(w, count=warm)
    cap = capture_step(oracle, w, body_cap=30000, contact_cap=80000)
    oracle.destroy(w)
    if scene == "plank":
        assert cap["colorStart"][12] > cap["colorStart"][11]
    cap = _spread(cap, stride)
    states, manifolds = solve_on_device(gpu, torch, cap)
    assert np.array_equal(states.view(np.uint32), cap["statesOut"].view(np.uint32))
    assert np.array_equal(manifolds, cap["manifoldsOut"])


def _tile(cap, copies):
    """The same set `copies` times over, side by side."""
    n = len(cap["statesIn"])
    starts = cap["colorStart"]
    out = dict(cap)
    for k in ("statesIn", "statesOut", "mass", "force", "damping"):
        out[k] = np.concatenate([cap[k]] * copies)
    out["awake"] = np.concatenate([cap["awake"] + i * n for i in range(copies)]).astype(np.int32)
    order = np.concatenate([np.arange(a, b) for a, b in zip(starts[:12], starts[1:13]) for _ in range(copies)])
    shift = np.concatenate([np.full(b - a, i * n) for a, b in zip(starts[:12], starts[1:13]) for i in range(copies)])
    bodies = cap["contactBodies"][order]
    out["contactBodies"] = np.where(bodies < 0, -1, bodies + shift[:, None]).astype(np.int32)
    out["mix"] = cap["mix"][order]
    for k in ("manifoldsIn", "manifoldsOut"):
        out[k] = cap[k].reshape(starts[12], -1)[order].reshape(-1)
    out["colorStart"] = [copies * c for c in starts]
    return out


# a grid's rows in shared memory, and in the row arrays when a CTA's share does not fit
# (about 240000 contacts)
@pytest.mark.gpu
@pytest.mark.parametrize("copies", [2, 5])
def test_resident_solver_large_sets(gpu, oracle, copies):
    torch = pytest.importorskip("torch")
    w, warm = _scene(oracle, "many")
    oracle.step(w, count=warm)
    cap = capture_step(oracle, w, body_cap=30000, contact_cap=80000)
    oracle.destroy(w)
    cap = _tile(cap, copies)
    assert (len(cap["contactBodies"]) > 250000) == (copies == 5)
    states, manifolds = solve_on_device(gpu, torch, cap)
    assert np.array_equal(states.view(np.uint32), cap["statesOut"].view(np.uint32))
    assert np.array_equal(manifolds, cap["manifoldsOut"])


# contacts in random order within their colours: a cluster's CTAs touch bodies of all
# others, and their copies fit (60) or do not (100)
@pytest.mark.gpu
@pytest.mark.parametrize("scene,stride", [("60", 1), ("100", 1), ("100", 3)])
def test_resident_solver_mixed_order(gpu, oracle, scene, stride):
    torch = pytest.importorskip("torch")
    w, warm = _scene(oracle, scene)
    oracle.step(w, count=warm)
    cap = capture_step(oracle, w)
    oracle.destroy(w)
    rng = np.random.default_rng(3)
    starts = cap["colorStart"]
    order = np.concatenate([rng.permutation(np.arange(a, b)) for a, b in zip(starts[:11], starts[1:12])]
                           + [np.arange(starts[11], starts[12])]).astype(np.int64)
    assert len(order) == len(cap["contactBodies"])
    for k in ("contactBodies", "mix"):
        cap[k] = cap[k][order]
    for k in ("manifoldsIn", "manifoldsOut"):
        cap[k] = cap[k].reshape(len(order), -1)[order].reshape(-1)
    cap = _spread(cap, stride)
    states, manifolds = solve_on_device(gpu, torch, cap)
    assert np.array_equal(states.view(np.uint32), cap["statesOut"].view(np.uint32))
    assert np.array_equal(manifolds, cap["manifoldsOut"])


@pytest.mark.gpu
def test_resident_solver_captured(gpu, oracle):
    """Both entry points inside a stream capture, replayed twice on the same inputs."""
    torch = pytest.importorskip("torch")
    bind_solve_api(gpu.lib)
    gpu.lib.b2SolveContactsNoAlloc.argtypes = gpu.lib.b2SolveContacts.argtypes
    gpu.lib.b2SolveContactsNoAlloc.restype = C.c_int
    for size, names in ((21, ("b2SolveContacts", "b2SolveContactsNoAlloc")), (120, ("b2SolveContacts",))):
        w, warm = _scene(oracle, str(size))
        oracle.step(w, count=warm)
        cap = capture_step(oracle, w)
        oracle.destroy(w)
        for name in names:
            fn = getattr(gpu.lib, name)
            d, t = make_desc(torch, cap, "cuda:0")
            first = t["statesIn"].clone(), t["manifoldsIn"].clone()
            assert fn(C.byref(d)) == 0  # set-up outside the capture
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            s = torch.cuda.Stream()
            with torch.cuda.graph(g, stream=s):
                d.stream = s.cuda_stream
                assert fn(C.byref(d)) == 0
            for _ in range(2):
                t["statesIn"].copy_(first[0])
                t["manifoldsIn"].copy_(first[1])
                g.replay()
                torch.cuda.synchronize()
                assert np.array_equal(t["statesIn"].cpu().numpy().view(np.uint32), cap["statesOut"].view(np.uint32))
                assert np.array_equal(t["manifoldsIn"].cpu().numpy(), cap["manifoldsOut"])


# a world's stage: on both sides of what one CTA holds (rows and bodies of a pyramid of 31
# or 32 rows; records of the 760 or 840 joints of a grid), and joints that fit a cluster's
# shared memory (60) or not (100)
@pytest.mark.gpu
@pytest.mark.parametrize("scene,size,steps", [("pyramid", 2, 20), ("pyramid", 31, 25), ("pyramid", 32, 25), ("grid", 20, 25), ("grid", 21, 25),
                                              ("grid", 60, 8), ("grid", 100, 4)])
def test_world_stage_spaces(gpu, oracle, scene, size, steps):
    def make(b):
        return b.pyramid(size, 0.01, 3) if scene == "pyramid" else b.joint_grid(size, -10.0)

    bad, detail, _ = lockstep(gpu, oracle, make, steps, check_manifolds=True)
    assert bad is None, detail


# a cluster's body copies: they fit (100, 111), do not fit beside the rows (113), are not
# tried (115, 117), the world does not fit a cluster (119); bodies mixed over all CTAs,
# overflow rows and a joint (tumbler)
@pytest.mark.gpu
@pytest.mark.parametrize("scene,size,steps", [("pyramid", 100, 6), ("pyramid", 111, 3), ("pyramid", 113, 3), ("pyramid", 115, 3), ("pyramid", 117, 3),
                                              ("pyramid", 119, 3), ("tumbler", 1500, 40)])
def test_cluster_copies(gpu, oracle, scene, size, steps):
    def make(b):
        return b.pyramid(size, 0.01, 3) if scene == "pyramid" else b.tumbler(size, 5, 0)

    bad, detail, _ = lockstep(gpu, oracle, make, steps, check_manifolds=True)
    assert bad is None, detail


# worlds that one CTA does not hold, of islands that it does: rows, joints of every type
# and overflow sets in bins of islands, and steps with events in between, which run
# without them; then one island too large for a bin
@pytest.mark.gpu
@pytest.mark.parametrize("scene,steps", [("pyramids", 40), ("joints", 150), ("mixed", 40)])
def test_bins_of_islands(gpu, oracle_atan, scene, steps):
    def make(b):
        if scene == "joints":
            return b.joint_zoo(24, 0, 9)
        if scene == "pyramids":
            return b.many_pyramids(9, 7, 6)
        w = b.pyramid(34, 0.01, 3)  # the pyramid's island is too large for a bin
        for _ in range(40):
            b.scenes.b2s_add_square(w, 0.25)
        return w

    bad, detail, _ = lockstep(gpu, oracle_atan, make, steps, check_manifolds=True, check_islands=True)
    assert bad is None, detail


@pytest.mark.gpu
def test_read_back_follows_every_step(gpu, oracle):
    """Body states read back after each step, after several steps, after body edits and
    wakes, and after batched steps are the device's (a second world that is never read
    between steps, or the oracle, says what they are)."""
    from box2c_gb300.capi import Vec2, bind_batch_api, bind_gpu_api, world_array

    bind_gpu_api(gpu.lib)
    bind_batch_api(gpu.lib)

    def read(world):
        n = gpu.lib.b2World_GetBodyStates(world, None, 0)
        out = np.zeros((n, 7), np.float32)
        assert gpu.lib.b2World_GetBodyStates(world, out.ctypes.data, n) == n
        return out.view(np.uint32)

    scenes = [lambda b: b.pyramid(8, 0.01, 3), lambda b: b.fast_shots(20), lambda b: b.sleep_scene(), lambda b: b.tumbler(80, 5, 0)]
    for k, make in enumerate(scenes):
        w, o = make(gpu), make(oracle)
        for step in range(1, 150 if k == 2 else 90):
            batched = step % 5 == 0 and k != 2
            if batched:
                ids = world_array([w])
                gpu.lib.b2World_StepBatch(ids, 1, 1.0 / 60.0, 4)
            else:
                gpu.step(w)
            oracle.step(o)
            if k == 2:  # scripted wakes, destructions and velocity changes
                gpu.sleep_step(w, step)
                oracle.sleep_step(o, step)
            if step % 7 in (0, 1, 2):
                got = read(w).view(np.float32)
                want = oracle.bodies(o)[:, :7]
                live = np.isfinite(want).all(1)
                cols = 4 if k == 2 else 7  # a sleeping body keeps its last velocity here
                assert np.array_equal(got[live][:, :cols].view(np.uint32), want[live][:, :cols].view(np.uint32)), (k, step)
                # a second read is the same, and so is one of the full mirror
                assert np.array_equal(read(w), got.view(np.uint32))
                full = gpu.bodies(w)[:, :7]
                both = np.isfinite(full).all(1)
                assert np.array_equal(got[both][:, :4].view(np.uint32), full[both][:, :4].view(np.uint32)), (k, step)
        gpu.destroy(w)
        oracle.destroy(o)


@pytest.mark.gpu
def test_batched_rows_beside_the_chip(gpu, oracle):
    """Batched worlds whose rows fit their group's shared memory, fit it in part (pyramids
    of 30 rows and more; overflow rows and a joint in the tumbler) and lie in it alone, over
    every launch shape the first steps try.  Tolerance: none."""
    from box2c_gb300.capi import bind_batch_api, world_array

    bind_batch_api(gpu.lib)

    def make(b):
        return [b.pyramid(n, 0.01, 3) for n in (2, 12, 20, 29, 30, 31, 38, 45)] + [b.tumbler(900, 5, 0)]

    batch, alone = make(gpu), make(oracle)
    ids = world_array(batch)
    for step in range(24):
        gpu.lib.b2World_StepBatch(ids, len(batch), 1.0 / 60.0, 4)
        for w in alone:
            oracle.step(w)
    for i, (w, o) in enumerate(zip(batch, alone)):
        got, want = gpu.bodies(w)[:, :7], oracle.bodies(o)[:, :7]
        live = np.isfinite(want).all(1)
        assert np.array_equal(got[live].view(np.uint32), want[live].view(np.uint32)), i
        gpu.destroy(w)
        oracle.destroy(o)


# bodies that contacts touch and the list leaves out: kinematic shelves at rest, whose
# integration changes nothing, so that the oracle's step is the expected result.  One CTA
# (8 shelves), a cluster (80, 120) with the contacts of the shelves spread over CTAs that do not
# own them, CTA 0 held up by an overflow set (wide shelves of 16), and a grid with its rows in memory (1000).
# Tolerance: none but the sign of a zero.
@pytest.mark.gpu
@pytest.mark.parametrize("shelves,wide,narrow", [(8, 8, 4), (8, 16, 8), (120, 8, 5), (80, 16, 8), (1000, 16, 8)])
def test_resident_solver_unlisted_bodies(gpu, oracle, shelves, wide, narrow):
    torch = pytest.importorskip("torch")
    w = oracle.shelves(shelves, wide, narrow)
    oracle.step(w, count=12)
    cap = capture_step(oracle, w, body_cap=30000, contact_cap=80000)
    oracle.destroy(w)
    kinematic = cap["mass"][cap["awake"], 1] == 0
    assert kinematic.sum() == shelves and (cap["colorStart"][12] > cap["colorStart"][11]) == (wide > 11)
    # the narrow shelves, whose contacts are the last of their colours, first
    n = len(cap["statesIn"])
    shelf = np.sort(cap["awake"][kinematic])
    order = np.concatenate([shelf[1::2], np.setdiff1d(np.arange(n), shelf[1::2])])
    place = np.empty(n, np.int32)
    place[order] = np.arange(n)
    for k in ("statesIn", "statesOut", "mass", "force", "damping"):
        cap[k] = cap[k][order]
    cap["contactBodies"] = np.where(cap["contactBodies"] < 0, -1, place[cap["contactBodies"]]).astype(np.int32)
    rng = np.random.default_rng(11)
    for drop in (kinematic, kinematic & (rng.random(len(kinematic)) < 0.5)):
        part = dict(cap, awake=place[cap["awake"][~drop]])
        states, manifolds = solve_on_device(gpu, torch, part)
        assert np.array_equal(states, cap["statesOut"])
        got, want = manifolds.view(np.float32), cap["manifoldsOut"].view(np.float32)
        assert np.all((got == want) | (got.view(np.uint32) == want.view(np.uint32)))


@pytest.mark.gpu
def test_solve_that_gives_up_is_marked(tmp_path):
    """A cluster or grid whose waits run out (tests/cuda/give_up_check.cu, compiled with limits
    of one poll) writes NaN velocities of all listed bodies."""
    here = os.path.dirname(os.path.abspath(__file__))
    src = os.path.join(os.path.dirname(here), "box2c_gb300", "csrc")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    flags = ["-gencode", "arch=compute_103a,code=sm_103a", "-O2", "--fmad=false", "-std=c++17", "-DPUSH_SPIN_LIMIT=1", "-DRES_SPIN_LIMIT=1",
             "-I", os.path.join(os.path.dirname(here), "include"), "-I", src]
    exe = str(tmp_path / "give_up_check")
    files = ["solve_api.cu", "resident.cu", "kernels.cu", "fused.cu", "arena.cu", "util.c"]
    subprocess.run([nvcc, "-t", "0", *flags, os.path.join(here, "cuda", "give_up_check.cu"), *[os.path.join(src, f) for f in files], "-o", exe],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "MISMATCH" not in r.stdout and "status no error" in r.stdout


def _slots(starts, ctas):
    """Body slots that the rows of a set without overflow leave a CTA of 226 KB."""
    rows = sum(-(-(b - a) // ctas) for a, b in zip(starts[:11], starts[1:12]))
    return (226 * 1024 - 144 * rows) // 60


# sets with as many listed bodies as a space holds beside their rows, and a few fewer and
# more: the contacts of a pyramid with bodies in free fall added, one CTA and a cluster
@pytest.mark.gpu
@pytest.mark.parametrize("scene,ctas", [("21", 1), ("24", 1), ("27", 1), ("60", 16), ("100", 16), ("105", 16)])
def test_resident_solver_body_edges(gpu, oracle, scene, ctas):
    torch = pytest.importorskip("torch")
    w, warm = _scene(oracle, scene)
    oracle.step(w, count=warm)
    cap = capture_step(oracle, w)
    oracle.destroy(w)
    w = oracle.drop_boxes(np.array([9.0], np.float32), np.array([0.5]), np.array([-1.0]), 0.6)
    free = capture_step(oracle, w)
    oracle.destroy(w)
    one = free["awake"][0]
    assert len(free["awake"]) == 1 and len(free["contactBodies"]) == 0
    edge = _slots(cap["colorStart"], ctas)
    n, listed = len(cap["statesIn"]), len(cap["awake"])
    for slots in range(edge - 4, edge + 2):
        for bodies in {ctas * slots - ctas + 1, ctas * slots}:
            more = bodies - listed
            assert more > 0
            part = dict(cap)
            for k in ("statesIn", "statesOut", "mass", "force", "damping"):
                part[k] = np.concatenate([cap[k], np.repeat(free[k][one:one + 1], more, axis=0)])
            part["awake"] = np.concatenate([cap["awake"], n + np.arange(more)]).astype(np.int32)
            states, manifolds = solve_on_device(gpu, torch, part)
            assert np.array_equal(states.view(np.uint32), part["statesOut"].view(np.uint32)), (slots, bodies)
            assert np.array_equal(manifolds, cap["manifoldsOut"]), (slots, bodies)


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [False, True])
def test_bytes_of_read_back_states(gpu, batched):
    """A step of a world that is read counts the 48 bytes a body that it writes to the host."""
    from box2c_gb300.capi import bind_batch_api, bind_gpu_api, world_array

    bind_gpu_api(gpu.lib)
    bind_batch_api(gpu.lib)
    w = gpu.pyramid(12, 0.0, 1)
    ids = world_array([w])

    def moved():
        if batched:
            gpu.lib.b2World_StepBatch(ids, 1, 1.0 / 60.0, 4)
        else:
            gpu.step(w)
        return gpu.lib.b2World_GetDeviceTimes(w).deviceToHostBytes

    for _ in range(40):
        before = moved()
    n = gpu.lib.b2World_GetBodyStates(w, None, 0)
    out = np.zeros((n, 7), np.float32)
    gpu.lib.b2World_GetBodyStates(w, out.ctypes.data, n)
    times = gpu.lib.b2World_GetDeviceTimes(w)
    after = moved()
    grown = 48 * (gpu.lib.b2World_GetDeviceTimes(w).recordCount - times.recordCount)
    assert after - before == 48 * 78 + grown
    gpu.destroy(w)
