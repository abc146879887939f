"""Env steps of one launch: what shared memory carries from step to step -- near
sets, consumed forces, broken grips, multipliers -- against launches of one
step each and against the f32 oracle, and that the worlds of
test_gpu_units.py's collision tests do collide."""
import ctypes as C

import numpy as np
import pytest

from kraken_3_gpu_b200 import _native
from oracle import binding as ob
from test_gpu_units import _F32P, _U32P, RECTS, _blocks, _clutter, _run

pytestmark = pytest.mark.gpu


def _chains(seed, brk=1e9):
    """Six chains of seven bodies with two points each among small rects, five
    of them flying at 300 px/s; grips at some ends, the resting one's with a
    break force of brk."""
    r = np.random.default_rng(seed)
    o = ob.World()
    o.set_rects(_clutter(20, seed))
    for k in range(6):
        x, y = 60 + 50 * k, r.uniform(60, 220)
        v = r.uniform(-1, 1, 2)
        v *= (0 if k == 3 else 300) / np.hypot(*v)
        for j in range(7):
            b = o.add_body(x, y + 9 * j, np.pi / 2, r.uniform(2, 6), r.uniform(60, 200))
            o.arr("vx")[b], o.arr("vy")[b] = v
            for e in (-4.0, 4.0):
                o.add_collision_point(b, e, 0.0, 3.0)
            if j:
                o.add_constraint(0, b - 1, b, 4.5, 0, -4.5, 0, 0.0)
                c = o.add_constraint(1, b - 1, b, 0, 0, 0, 0, 1e-6)
                c.target, c.minAngle, c.maxAngle = r.uniform(-0.4, 0.4), -1.0, 1.0
        if k % 2:
            c = o.add_constraint(2, b, -1, 4.5, 0, x, y + 58.5, 0.0)
            c.breakForce = brk if k == 3 else 1e9
    o.set_list(np.arange(o.nC))
    o.f32ify()
    o.round_state()
    return o


def _break_midway(seed, steps):
    """A break force that the resting chain's grip first exceeds after the
    first step, and the force field."""
    o = _chains(seed)
    force = np.random.default_rng(seed).uniform(-400, 400, (o.n, 3)).astype(np.float32)
    for f, k in (("fx", 0), ("fy", 1), ("tq", 2)):
        o.arr(f)[:] = force[:, k]
    grip = [c for c in o.constraints if c.type == 2][1]
    pull = []
    for _ in range(steps):
        o.step32()
        pull.append(120 * np.hypot(grip.lambdaX, grip.lambdaY))
    s = next(s for s in range(1, steps) if pull[s] > max(pull[:s]))
    return 0.5 * (pull[s] + max(pull[:s])), force


@pytest.mark.parametrize("seed,steps", [(1, 40), (2, 128), (3, 129), (6, 300)])
def test_steps_of_one_call_equal_single_steps_and_the_oracle(seed, steps):
    brk, force = _break_midway(seed, steps)
    o = _chains(seed, brk)
    bodies, cons, pts, rng, forces = _blocks(o, force)
    rects = _clutter(20, seed).astype(np.float32)
    start = bodies[:, :2].copy()
    L = _native.lib()
    p = _native.SolverParams(1 / 120, 2, 4, 3.0, 3.0, 360.0, 18.0)
    out = []
    for calls in ([steps], [1] * steps):
        h = C.c_void_p()
        b, c = bodies.copy(), cons.copy()
        _native.check(L.kr_create(C.byref(p), o.n, o.nC, rects.ctypes.data_as(_F32P), len(rects),
                                  pts.ctypes.data_as(_U32P), len(pts), rng.ctypes.data_as(_U32P), C.byref(h)))
        try:
            _native.check(L.kr_upload(h, b.ctypes.data_as(_F32P), c.ctypes.data_as(_U32P),
                                      forces.ctypes.data_as(_F32P), None), h)
            for k in calls:
                _native.check(L.kr_step(h, k), h)
            _native.check(L.kr_download(h, b.ctypes.data_as(_F32P), c.ctypes.data_as(_U32P)), h)
        finally:
            L.kr_destroy(h)
        out.append((b, c))
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(*out))
    for f, k in (("fx", 0), ("fy", 1), ("tq", 2)):
        o.arr(f)[:] = force[:, k]
    hits, broke = 0, []
    for s in range(steps):
        o.step32()
        hits += o.stats["collisions"]
        broke += [s for c in o.constraints if c.broken]
    got = out[0][0]
    for c, f in ((0, "px"), (1, "py"), (4, "vx"), (5, "vy"), (6, "ang"), (8, "av")):
        assert np.array_equal(got[:, c], o.arr(f).astype(np.float32)), f
    assert [bool(v) for v in out[0][1].view(np.uint32)[:, 17]] == [bool(c.broken) for c in o.constraints]
    # the run has what it is for: walls, bodies beyond any collision reference's
    # 32 px of where they started, a grip that broke on the way
    assert hits > 100 and np.abs(got[:, :2] - start).max() > 32
    assert broke and broke[0] > 0 and len({c.broken for c in o.constraints}) == 2


@pytest.mark.parametrize("n,offset", [(0, 0.0), (12, 0.0), (27, 0.0), (58, 0.0), (200, 0.0), (12, 31900.0),
                                      (12, 40000.0), (200, -300000.0)])
def test_the_collision_worlds_collide(n, offset):
    rects = _clutter(n, n) + np.array([offset, offset, 0, 0])
    assert sum(_run(100 + seed, 14, 10, 200, rects, offset) for seed in range(4)) > 100
