"""Handles over their lifetime: what closing one gives back, and an upload
that replaces a world while its steps are in flight."""
import ctypes as C

import numpy as np
import pytest

from kraken_3_gpu_b200 import _native, batch
from oracle import binding as ob

pytestmark = pytest.mark.gpu

_F32P, _U32P = C.POINTER(C.c_float), C.POINTER(C.c_uint32)
PARAMS = _native.SolverParams(1 / 120, 2, 4, 3.0, 3.0, 360.0, 18.0)
RECTS = np.array([[0, 0, 400, 14], [0, 286, 400, 14], [0, 0, 14, 300], [386, 0, 14, 300]], np.float32)


def _world(n, nc):
    """A drop-in handle of n bodies without collision points and nc constraints."""
    h = C.c_void_p()
    _native.check(_native.lib().kr_create(C.byref(PARAMS), n, nc, RECTS.ctypes.data_as(_F32P), len(RECTS), None, 0,
                                          None, C.byref(h)))
    return h


def _bodies(n, seed):
    r = np.random.default_rng(seed)
    b = np.zeros((n, 12), np.float32)
    b[:, 0], b[:, 1], b[:, 6] = r.uniform(30, 350, n), r.uniform(30, 250, n), r.uniform(-3, 3, n)
    b[:, 2:4], b[:, 7] = b[:, :2], b[:, 6]
    b[:, 9], b[:, 10] = 1 / r.uniform(1, 20, n), 1 / r.uniform(20, 900, n)
    return b


def _chains(n, size):
    """Pin and angle constraints along chains of `size` bodies out of n, as
    many records as 2 n (the last ones pin single bodies to the world)."""
    cons = np.zeros((2 * n, 20), np.float32)
    cu = cons.view(np.uint32)
    k = 0
    for i in range(n):
        if i % size != size - 1:
            for t in (0, 1):
                cu[k, 0], cu[k, 1], cu[k, 2] = i, i + 1, t
                k += 1
    for i in range(2 * n - k):
        cu[k, 0], cu[k, 1], cu[k, 2] = i % n, 0xFFFFFFFF, 0
        cons[k, 6:8] = 100 + i % 90
        k += 1
    cons[:, 4], cons[:, 8] = 6.0, 1e-5
    cons[:, 11], cons[:, 12], cons[:, 16] = -1, 1, 400
    return cons


def _upload(h, bodies, cons):
    _native.check(_native.lib().kr_upload(h, bodies.ctypes.data_as(_F32P), cons.ctypes.data_as(_U32P), None, None), h)


def _step(h, steps):
    _native.check(_native.lib().kr_step(h, steps), h)


def _download(h, n, nc):
    bodies, cons = np.zeros((n, 12), np.float32), np.zeros((nc, 20), np.float32)
    _native.check(_native.lib().kr_download(h, bodies.ctypes.data_as(_F32P), cons.ctypes.data_as(_U32P)), h)
    return bodies.view(np.uint32), cons.view(np.uint32)


def _free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_closed_engines_give_their_memory_back():
    """An engine of 16,384 one-segment creatures holds 64 KB of launch groups
    and its queue word: 300 engines that ran and were closed must leave the
    device's free memory as the first ten left it (21 MB less when the groups
    stay behind; the driver hands out small blocks 2 MB at a time)."""
    n = 16384
    x = np.full(n, 400.0)
    maps = [ob.make_map_rects(seed=1)]

    def one():
        eng = batch.BatchEngine(maps, n)
        eng.spawn(0, np.ones(n, int), np.ones(n, int), np.zeros(n, int), x, x, np.zeros(n), np.ones(n, int))
        eng.run(1)
        eng.sync()
        eng.close()

    for _ in range(10):
        one()
    before = _free_bytes()
    for _ in range(300):
        one()
    assert before - _free_bytes() < 4 << 20


@pytest.mark.parametrize("size", [(40, 3), (2, 48)])
def test_upload_during_steps_equals_a_fresh_handle(size):
    """kr_step returns while its launches (of up to 128 env steps each) run;
    an upload of another constraint structure right behind it replaces the
    tables that they read, and must wait for them."""
    n = 1920
    first, second = _chains(n, size[0]), _chains(n, size[1])
    a, b = _world(n, 2 * n), _world(n, 2 * n)
    try:
        for turn in range(3):
            _upload(a, _bodies(n, 1), first)
            _step(a, 300)
            _upload(a, _bodies(n, 2 + turn), second)
            _step(a, 20)
            got = _download(a, n, 2 * n)
            _upload(b, _bodies(n, 2 + turn), second)
            _step(b, 20)
            want = _download(b, n, 2 * n)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        for h in (a, b):
            _native.lib().kr_destroy(h)


@pytest.mark.parametrize("nb,nc", [(40, 150), (160, 384)])
def test_handles_of_unlike_islands_step_side_by_side(nb, nc):
    """A handle whose island needs more shared memory than a launch has by
    default, then the upload of a small one: both step, in either order, to
    what each gives by itself."""
    cons = np.zeros((nc, 20), np.float32)
    cu = cons.view(np.uint32)
    for k in range(nc):
        cu[k, 0], cu[k, 1] = (k, k + 1) if k < nb - 1 else (k % nb, 0xFFFFFFFF)
    cons[nb - 1:, 6:8] = 150
    cons[:, 4], cons[:, 8], cons[:, 16] = 6.0, 1e-5, 400
    order = np.concatenate([np.arange(0, nb - 1, 2), np.arange(1, nb - 1, 2), np.arange(nb - 1, nc)])
    cons = cons[order]
    L = _native.lib()
    alone = []
    for n, c in ((nb, cons), (2, _chains(2, 2))):
        h = _world(n, len(c))
        _upload(h, _bodies(n, 5), c)
        _step(h, 3)
        alone.append(_download(h, n, len(c)))
        L.kr_destroy(h)
    a, b = _world(nb, nc), _world(2, 4)
    try:
        _upload(a, _bodies(nb, 5), cons)
        _upload(b, _bodies(2, 5), _chains(2, 2))
        _step(a, 3)
        _step(b, 3)
        for got, want in ((_download(a, nb, nc), alone[0]), (_download(b, 2, 4), alone[1])):
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        for h in (a, b):
            L.kr_destroy(h)


# the launch shapes in whose share of an SM's shared memory a creature fits at a
# word per field: by body, lanes, warps and CTAs per SM (0: 16 / warps), taken or not
SHAPES = [(6, 7, 32, 1, 0, True), (6, 7, 32, 1, 16, True), (6, 7, 32, 1, 17, True), (6, 7, 32, 1, 19, False),
          (6, 7, 16, 1, 16, True), (4, 5, 32, 1, 16, True), (8, 9, 32, 2, 0, True), (8, 9, 32, 1, 0, False),
          (8, 9, 8, 16, 1, True), (1, 1, 32, 1, 32, True), (2, 2, 8, 2, 32, True)]


@pytest.mark.parametrize("arms,segs,lanes,warps,ctas,taken", SHAPES)
def test_launch_shapes_taken_and_refused(arms, segs, lanes, warps, ctas, taken):
    """What kr_batch_set_launch takes runs, with the automatic shape's results,
    also where the kernel's records need more than the shape's share of the
    shared memory; what is too large for it is refused when it runs."""
    n = 70
    r = np.random.default_rng(3)
    args = (np.full(n, arms), np.full(n, segs), np.zeros(n, int), r.uniform(300, 1000, n), r.uniform(300, 500, n),
            r.uniform(0, 6, n), r.integers(5, 20, n))
    out = []
    for shape in (None, (warps, ctas, lanes)):
        eng = batch.BatchEngine([ob.make_map_rects(seed=3)], n)
        eng.spawn(0, *args)
        if shape:
            eng.set_launch(shape[0], shape[1], lanes_per_creature=shape[2])
        if shape and not taken:
            with pytest.raises(_native.KrError) as e:
                eng.run(20)
            assert e.value.code == _native.KR_ERR_CAPACITY
        else:
            eng.run(20)
            out.append(eng.read_state())
        eng.close()
    if taken:
        assert all(np.array_equal(out[0][f], out[1][f]) for f in out[0])


def test_engines_of_two_threads_launch_side_by_side():
    """Two engines whose CTAs need unlike amounts of shared memory, each driven
    by a thread of its own: every launch goes through, and to the state that
    each engine reaches by itself."""
    from concurrent.futures import ThreadPoolExecutor

    maps = [ob.make_map_rects(seed=3)]

    def engine(arms, segs, n):
        r = np.random.default_rng(arms)
        eng = batch.BatchEngine(maps, n)
        eng.spawn(0, np.full(n, arms), np.full(n, segs), np.zeros(n, int), r.uniform(300, 1000, n),
                  r.uniform(300, 500, n), r.uniform(0, 6, n), np.full(n, 400))
        return eng

    def drive(eng):
        for _ in range(400):
            eng.run(1)
        return eng.read_state()

    shapes = ((8, 9, 6), (1, 1, 6))
    alone = []
    for s in shapes:
        eng = engine(*s)
        alone.append(drive(eng))
        eng.close()
    engines = [engine(*s) for s in shapes]
    with ThreadPoolExecutor(2) as pool:
        got = list(pool.map(drive, engines))
    for a, g in zip(alone, got):
        assert all(np.array_equal(a[f], g[f]) for f in a)
    for eng in engines:
        eng.close()
