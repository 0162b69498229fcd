"""The backward pass gives a world the same gradient, bit for bit, whichever way it runs:
rows in lanes' registers (at most 32 rows), replays in shared memory, replays in global
memory (large worlds), all steps in one chunk or in several."""
import numpy as np
import pytest

from box2c_gb300.autograd import bind_adjoint_api
from box2c_gb300.capi import bind_batch_api, bind_gpu_api, world_array

pytestmark = pytest.mark.gpu
STEPS = 40


def _drop(gpu):
    kinds = np.array([0, 1, 2, 0, 1, 2, 0, 0], np.int32)
    h = np.array([0.6, 0.7, 0.8, 1.7, 1.9, 2.0, 2.7, 2.9], np.float32)
    return gpu.drop_boxes(h, np.linspace(-1, 1, 8), np.linspace(1, -1, 8), 0.5, kinds)


def _plank(gpu):
    n = 17
    kinds = np.array([3] + [0] * (n - 1), np.int32)
    h = np.array([0.2] + [0.9 + 0.01 * (k % 3) for k in range(n - 1)], np.float32)
    return gpu.drop_boxes(h, np.linspace(-0.1, 0.1, n), np.zeros(n), 0.6, kinds)


def _stack(gpu):
    return gpu.pyramid(6, 0.01, 3)


def _pile(gpu):
    return gpu.pyramid(14, 0.01, 4)


def _record(gpu, makers, steps=STEPS):
    worlds = [m(gpu) for m in makers]
    for w in worlds:
        gpu.lib.b2World_BeginTape(w, steps)
    ids = world_array(worlds)
    for _ in range(steps):
        gpu.lib.b2World_StepBatch(ids, len(worlds), 1.0 / 60.0, 4)
    return worlds


def _backward(gpu, worlds, seeds):
    sizes = [gpu.lib.b2World_GetBodyStates(w, None, 0) for w in worlds]
    stride = max(sizes)
    gf = np.zeros((len(worlds), stride, 6), np.float32)
    for i, (n, s) in enumerate(zip(sizes, seeds)):
        gf[i, :n] = np.random.default_rng(s).normal(0, 1, (n, 6))
    gi = np.zeros_like(gf)
    gm = np.zeros((len(worlds), stride), np.float32)
    rc = gpu.lib.b2World_StepBackwardBatch(world_array(worlds), len(worlds), stride, stride, gf.ctypes.data, gi.ctypes.data, gm.ctypes.data)
    assert rc == 0
    return [(gi[i, :n].copy().view(np.uint32), gm[i, :n].copy().view(np.uint32)) for i, n in enumerate(sizes)]


def test_backward_paths_agree(gpu):
    bind_gpu_api(gpu.lib)
    bind_batch_api(gpu.lib)
    bind_adjoint_api(gpu.lib)
    makers = [_drop, _plank, _stack, _pile]
    worlds = _record(gpu, makers)
    counts = [gpu.counters(w) for w in worlds]
    assert counts[1].colorCounts[11] > 0  # overflow rows
    rows = [sum(x.colorCounts) for x in counts]
    # one lane a row; shared memory; neither
    assert max(rows[0], rows[1]) <= 32 < rows[2] < 60 and rows[3] > 100
    alone = [_backward(gpu, [w], [k])[0] for k, w in enumerate(worlds)]
    assert all(np.isfinite(g.view(np.float32)).all() and (f != 0).any() for g, f in alone)
    for group in ([0, 1], [0, 2], [1, 2], [0, 3], [2, 3], [0, 1, 2, 3]):
        for got, k in zip(_backward(gpu, [worlds[k] for k in group], group), group):
            assert np.array_equal(got[0], alone[k][0]) and np.array_equal(got[1], alone[k][1]), (group, k)
    for w in worlds:
        gpu.destroy(w)


@pytest.mark.parametrize("maker,copies", [(_drop, 160), (_pile, 24)])
def test_backward_in_chunks(gpu, maker, copies):
    """Enough copies that the steps are replayed in several chunks."""
    bind_gpu_api(gpu.lib)
    bind_batch_api(gpu.lib)
    bind_adjoint_api(gpu.lib)
    steps = 110
    one = _record(gpu, [maker], steps)
    want = _backward(gpu, one, [5])[0]
    many = _record(gpu, [maker] * copies, steps)
    for got in _backward(gpu, many, [5] * copies):
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    for w in one + many:
        gpu.destroy(w)


def test_backward_of_many_worlds(gpu):
    """More worlds than a grid's second dimension holds, each without a recorded step: the
    kernels are launched and do nothing."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    launch = gpu.lib.b2gd_adjoint_launch
    launch.argtypes = [C.c_void_p] + [C.c_int] * 6 + [C.c_void_p]
    launch.restype = C.c_int
    worlds = 70000
    items = torch.zeros(worlds * 4096, dtype=torch.uint8, device="cuda:0")  # an item is smaller
    torch.cuda.synchronize()
    assert launch(items.data_ptr(), worlds, 1, 1, 1, 1, 4, None) == 0
    torch.cuda.synchronize()
    assert not items.any()
