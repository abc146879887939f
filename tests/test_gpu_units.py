"""The drop-in's solve units against the f32 oracle's sequential sweep, on
worlds no creature looks like: random constraint lists with repeated and
reversed pairs, both bodies the same, angle constraints against the world,
pins with compliance, grips between bodies, broken flags on every type,
immovable bodies, forces, and passes of more than 32 units.  The oracle solves
the list constraint by constraint; the kernel solves units in passes, the same
operations per body in the same order, so every value must be equal -- up to
the step in which a world that tears itself apart throws a body beyond 1e6 px
(angles then jump by more than the f32 quotient of the angle wrap covers)."""
import ctypes as C

import numpy as np
import pytest

from kraken_3_gpu_b200 import _native, batch
from oracle import binding as ob

pytestmark = pytest.mark.gpu

_F32P, _U32P = C.POINTER(C.c_float), C.POINTER(C.c_uint32)
RECTS = np.array([[0, 0, 400, 14], [0, 286, 400, 14], [0, 0, 14, 300], [386, 0, 14, 300], [150, 120, 90, 18]], float)


def _random_world(seed, nb, nc, spread, rects=RECTS, offset=0.0):
    r = np.random.default_rng(seed)
    o = ob.World()
    o.set_rects(rects)
    for i in range(nb):
        fixed = r.random() < 0.1
        o.add_body(offset + r.uniform(30, 30 + spread), offset + r.uniform(30, 30 + 0.6 * spread), r.uniform(-7, 7),
                   0 if fixed else r.uniform(1, 20), 0 if fixed and r.random() < 0.5 else r.uniform(20, 900))
        for _ in range(int(r.integers(0, 4))):
            o.add_collision_point(i, r.uniform(-8, 8), r.uniform(-8, 8), r.uniform(2, 7))
    pair = (0, -1)
    for k in range(nc):
        if r.random() < 0.6 or k == 0:
            a = int(r.integers(nb))
            b = -1 if r.random() < 0.2 else int(r.integers(nb))
            if b == a and r.random() < 0.5:
                b = -1
            pair = (a, b)
        elif pair[1] >= 0 and r.random() < 0.2:
            pair = pair[::-1]
        a, b = pair
        t = int(r.integers(3))
        c = o.add_constraint(t, a, b, r.uniform(-7, 7), r.uniform(-7, 7),
                             offset + r.uniform(40, 200) if b < 0 else r.uniform(-7, 7),
                             offset + r.uniform(40, 150) if b < 0 else r.uniform(-7, 7),
                             r.choice([0.0, 1e-6, 1e-5]))
        c.rest, c.target = r.uniform(-3, 3), r.uniform(-1, 1)
        c.minAngle, c.maxAngle = -r.uniform(0.1, 2), r.uniform(0.1, 2)
        c.broken = r.random() < 0.15
        c.breakForce = r.uniform(5, 400)
    o.set_list(np.arange(nc))
    o.f32ify()
    o.round_state()
    return o, r.uniform(-400, 400, (nb, 3)).astype(np.float32)


def _blocks(o, force):
    bodies = np.zeros((o.n, 12), np.float32)
    for c, f in enumerate(("px", "py", "ppx", "ppy", "vx", "vy", "ang", "angP", "av", "im", "ii")):
        bodies[:, c] = o.arr(f)
    cons = np.zeros((o.nC, 20), np.float32)
    cu = cons.view(np.uint32)
    for k, c in enumerate(o.constraints):
        cu[k, 0], cu[k, 1], cu[k, 2] = c.a, c.b & 0xFFFFFFFF, c.type
        cons[k, 4:13] = (c.lax, c.lay, c.lbx, c.lby, c.compliance, c.rest, c.target, c.minAngle, c.maxAngle)
        cons[k, 16] = c.breakForce
        cu[k, 17] = c.broken
    pts = np.array(o.coll_pts(), np.float32).reshape(-1, 4)
    body = pts[:, 0].astype(np.int64)
    order = np.argsort(body, kind="stable")
    pts, body = np.ascontiguousarray(pts[order]), body[order]
    pts.view(np.uint32)[:, 0] = body
    cnt = np.bincount(body, minlength=o.n).astype(np.uint32)
    rng = np.concatenate([np.cumsum(cnt) - cnt, cnt]).astype(np.uint32)
    forces = np.zeros((o.n, 4), np.float32)
    forces[:, :3] = force
    return bodies, cons, pts, rng, forces


def _run(seed, nb, nc, spread, rects=RECTS, offset=0.0):
    o, force = _random_world(seed, nb, nc, spread, rects, offset)
    bodies, cons, pts, rng, forces = _blocks(o, force)
    L = _native.lib()
    h = C.c_void_p()
    p = _native.SolverParams(1 / 120, 2, 4, 3.0, 3.0, 360.0, 18.0)
    r32 = rects.astype(np.float32)
    _native.check(L.kr_create(C.byref(p), nb, nc, r32.ctypes.data_as(_F32P), len(r32), pts.ctypes.data_as(_U32P),
                              len(pts), rng.ctypes.data_as(_U32P), C.byref(h)))
    hits = 0
    try:
        cp = cons.ctypes.data_as(_U32P) if nc else None
        _native.check(L.kr_upload(h, bodies.ctypes.data_as(_F32P), cp, forces.ctypes.data_as(_F32P), None), h)
        for f, k in (("fx", 0), ("fy", 1), ("tq", 2)):
            o.arr(f)[:] = force[:, k]
        for s in range(12):
            _native.check(L.kr_step(h, 1), h)
            _native.check(L.kr_download(h, bodies.ctypes.data_as(_F32P), cp), h)
            o.step32()
            hits += o.stats["collisions"]
            if np.abs(o.arr("px")).max() > 1e6 or np.abs(o.arr("py")).max() > 1e6:
                assert s >= 2
                break
            for c, f in ((0, "px"), (1, "py"), (4, "vx"), (5, "vy"), (6, "ang"), (8, "av")):
                assert np.array_equal(bodies[:, c], o.arr(f).astype(np.float32)), (s, f)
            for k, c in enumerate(o.constraints):
                lam = (cons[k, 15],) if c.type == 1 else (cons[k, 13], cons[k, 14])
                ref = (getattr(c, "lambda"),) if c.type == 1 else (c.lambdaX, c.lambdaY)
                assert tuple(np.float32(v) for v in ref) == tuple(lam), (s, k)
                assert bool(cons.view(np.uint32)[k, 17]) == c.broken, (s, k)
    finally:
        L.kr_destroy(h)
    return hits


@pytest.mark.parametrize("seed,nb,nc,spread", [(s, 12, 40, 160) for s in range(8)] + [(8, 2, 6, 20), (9, 1, 3, 30),
                                                                                    (10, 90, 110, 300), (11, 5, 0, 60)])
def test_random_lists_equal_the_sequential_oracle(seed, nb, nc, spread):
    _run(seed, nb, nc, spread)


def _clutter(n, seed):
    """The walls and n small rects among the bodies."""
    r = np.random.default_rng(seed)
    return np.concatenate([RECTS, np.stack([r.uniform(20, 260, n), r.uniform(20, 200, n), r.uniform(4, 30, n),
                                            r.uniform(4, 30, n)], 1)])


@pytest.mark.parametrize("n,offset", [(0, 0.0), (12, 0.0), (25, 0.0), (26, 0.0), (27, 0.0), (40, 0.0), (56, 0.0),
                                      (57, 0.0), (58, 0.0), (200, 0.0),
                                      (70000, 0.0), (12, 31900.0), (12, 40000.0)])
def test_near_rects_equal_the_full_list(n, offset):
    """Collision passes over the near sets (one rect or two per mask bit), and
    over every rect where a creature has more than 62 near it, coordinates
    outside the references' range or the map more than 65,535 rects: the
    oracle folds over every rect each time."""
    rects = _clutter(min(n, 200), n)
    if n > 200:  # the rest far away, the near ones last
        far = np.tile([1e5, 1e5, 20.0, 20.0], (n - 200, 1))
        rects = np.concatenate([far, rects])
    rects = rects + np.array([offset, offset, 0, 0])
    for seed in range(2 if n > 200 else 4):
        _run(100 + seed, 14, 10, 200, rects, offset)


def test_angle_wrap_edges():
    """Pairs of bodies whose angle differences lie at the edges of the wrap:
    multiples of pi / 2 up to 8 pi, and where the near form ends, within a few
    ulp and on both sides."""
    o = ob.World()
    o.set_rects(RECTS)
    r = np.random.default_rng(3)
    edges = [k * np.pi / 2 for k in range(-16, 17)] + [9.42, -9.42, 4.0, -4.0, 49.9, -49.9]
    k = 0
    for e in edges:
        for d in (0.0, 3e-7, -3e-7, 2e-4, -2e-4, r.uniform(-0.3, 0.3)):
            for base in (0.0, r.uniform(-6, 6)):
                x, y = 20.0 + 5 * (k % 70), 20.0 + 5 * (k // 70)
                a = o.add_body(x, y, base, 2.0, 60.0)
                b = o.add_body(x, y, base + e + d, 3.0, 90.0)
                c = o.add_constraint(1, a, b, 0, 0, 0, 0, 1e-6 if k % 3 else 0.0)
                c.rest, c.target = (0.0, 0.0) if k % 2 else (r.uniform(0, 6.3), r.uniform(-1.9, 1.9))
                c.minAngle, c.maxAngle = -1.3, 1.3
                k += 1
    o.set_list(np.arange(o.nC))
    o.f32ify()
    o.round_state()
    bodies, cons, pts, rng, forces = _blocks(o, np.zeros((o.n, 3), np.float32))
    L = _native.lib()
    h = C.c_void_p()
    p = _native.SolverParams(1 / 120, 2, 4, 3.0, 3.0, 360.0, 18.0)
    r32 = RECTS.astype(np.float32)
    _native.check(L.kr_create(C.byref(p), o.n, o.nC, r32.ctypes.data_as(_F32P), len(r32), None, 0, None, C.byref(h)))
    try:
        cp = cons.ctypes.data_as(_U32P)
        _native.check(L.kr_upload(h, bodies.ctypes.data_as(_F32P), cp, None, None), h)
        for s in range(4):
            _native.check(L.kr_step(h, 1), h)
            _native.check(L.kr_download(h, bodies.ctypes.data_as(_F32P), cp), h)
            o.step32()
            assert np.array_equal(bodies[:, 6], o.arr("ang").astype(np.float32)), s
            assert np.array_equal(bodies[:, 8], o.arr("av").astype(np.float32)), s
    finally:
        L.kr_destroy(h)


def test_quotients_equal_ieee_division():
    """The shared-reciprocal quotients against IEEE f32 division: 1 / b for
    every mantissa of b, and quotients of random and extreme mantissas over
    the stated exponents.  (All 2^46 pairs of mantissas were compared once.)"""
    m = np.arange(1 << 23, dtype=np.uint32)
    b = (m | np.uint32(127 << 23)).view(np.float32)
    one = np.ones_like(b)
    assert np.array_equal(batch.probe_quot(one, b), one / b)
    r = np.random.default_rng(5)
    n = 1 << 21
    for ea, eb in ((0, 0), (59, -59), (-99, 59), (-60, -59), (20, -20), (-7, 3)):
        ma, mb = r.integers(0, 1 << 23, n), r.integers(0, 1 << 23, n)
        near = np.where(r.random(n // 2) < 0.5, r.integers(0, 8, n // 2), (1 << 23) - 1 - r.integers(0, 8, n // 2))
        ma[: n // 4], mb[n // 8: n // 2] = near[: n // 4], near[n // 8: n // 2]
        a = np.ldexp(1 + ma / 2.0 ** 23, ea).astype(np.float32) * r.choice([-1, 1], n).astype(np.float32)
        b = np.ldexp(1 + mb / 2.0 ** 23, eb).astype(np.float32)
        a[-1000:] = 0
        assert np.array_equal(batch.probe_quot(a, b), a / b), (ea, eb)


def _noalloc(L):
    L.kr_step_noalloc.restype = C.c_int
    L.kr_step_noalloc.argtypes = [C.POINTER(_native.SolverParams), C.c_uint32, C.c_uint32, C.c_void_p, C.c_void_p,
                                  C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_uint32, C.c_void_p, C.c_int32,
                                  C.c_void_p]
    return L


@pytest.mark.parametrize("islands,nb,nc,steps", [(1, 1, 1, 1), (1, 160, 384, 2), (33, 5, 9, 3), (300, 2, 3, 1),
                                                 (1024, 2, 4, 130), (2048, 1, 2, 1), (12, 160, 330, 2)])
def test_noalloc_schedule_equals_the_handles_step(islands, nb, nc, steps):
    """The allocation-free entry builds its schedule on the device: random
    islands whose bodies and constraints are shuffled among one another, from
    one body to the entry's limits, must step to the bytes that the handle's
    host-built schedule gives."""
    import torch

    r = np.random.default_rng(islands * 1000 + nb)
    n = islands * nb
    place = r.permutation(n)  # body (island, j) -> index
    bodies = np.zeros((n, 12), np.float32)
    bodies[:, 0], bodies[:, 1] = r.uniform(30, 350, n), r.uniform(30, 250, n)
    bodies[:, 2:4] = bodies[:, :2]
    bodies[:, 6] = bodies[:, 7] = r.uniform(-3, 3, n)
    bodies[:, 9], bodies[:, 10] = 1 / r.uniform(1, 20, n), 1 / r.uniform(20, 900, n)
    rows = []
    for i in range(islands):
        own = place[i * nb:(i + 1) * nb]
        level = np.zeros(nb, int)
        for k in range(nc):
            a = k % (nb - 1) if nb > 1 and k < nb - 1 else int(np.argmin(level))
            b = a + 1 if nb > 1 and k < nb - 1 else (-1 if nb == 1 or r.random() < 0.3 else int((a + 1 + r.integers(nb - 1)) % nb))
            t = int(r.integers(3))
            if b >= 0 and max(level[a], level[b]) > 80:
                b = -1
            level[a] = max(level[a], level[b] if b >= 0 else 0) + 1
            if b >= 0:
                level[b] = level[a]
            rows.append((i * nc + k, own[a], own[b] if b >= 0 else -1, t))
    order = np.argsort(r.random(len(rows)) * islands + np.array([q[0] % nc for q in rows]), kind="stable")
    cons = np.zeros((len(rows), 20), np.float32)
    cu = cons.view(np.uint32)
    for at, k in enumerate(order):
        _, a, b, t = rows[k]
        cu[at, 0], cu[at, 1], cu[at, 2] = a, b & 0xFFFFFFFF, t
        cons[at, 4:8] = r.uniform(-7, 7, 4)
        if b < 0:
            cons[at, 6:8] = r.uniform(40, 250, 2)
        cons[at, 8], cons[at, 9], cons[at, 10] = 1e-5, r.uniform(-1, 1), r.uniform(-1, 1)
        cons[at, 11], cons[at, 12], cons[at, 16] = -1, 1, r.uniform(50, 500)
    cnt = np.minimum(r.integers(0, 4, n), 4096 // n + 1).astype(np.uint32)
    while cnt.sum() > 4096:
        cnt[int(np.argmax(cnt))] -= 1
    rng = np.concatenate([np.cumsum(cnt) - cnt, cnt]).astype(np.uint32)
    pts = np.zeros((int(cnt.sum()), 4), np.float32)
    pts.view(np.uint32)[:, 0] = np.repeat(np.arange(n), cnt)
    pts[:, 1:3], pts[:, 3] = r.uniform(-6, 6, (len(pts), 2)), r.uniform(2, 7, len(pts))
    rects = RECTS.astype(np.float32)
    L = _noalloc(_native.lib())
    p = _native.SolverParams(1 / 120, 2, 4, 3.0, 3.0, 360.0, 18.0)
    dev = [torch.from_numpy(np.ascontiguousarray(v).view(np.int32)).cuda() for v in (bodies, cons, rects, pts, rng)]
    forces = torch.zeros((n, 4), device="cuda")
    args = (C.byref(p), n, len(cons), dev[0].data_ptr(), dev[1].data_ptr(), forces.data_ptr(), dev[2].data_ptr(),
            len(rects), dev[3].data_ptr(), len(pts), dev[4].data_ptr())
    rc = L.kr_step_noalloc(*args, steps, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    h = C.c_void_p()
    _native.check(L.kr_create(C.byref(p), n, len(cons), rects.ctypes.data_as(_F32P), len(rects),
                              pts.ctypes.data_as(_U32P), len(pts), rng.ctypes.data_as(_U32P), C.byref(h)))
    try:
        up = L.kr_upload(h, bodies.ctypes.data_as(_F32P), cu.ctypes.data_as(_U32P), None, None)
        assert rc == up
        if rc == 0:
            _native.check(L.kr_step(h, steps), h)
            _native.check(L.kr_download(h, bodies.ctypes.data_as(_F32P), cu.ctypes.data_as(_U32P)), h)
        assert np.array_equal(dev[0].cpu().numpy(), bodies.view(np.int32))
        assert np.array_equal(dev[1].cpu().numpy(), cons.view(np.int32))
    finally:
        L.kr_destroy(h)


@pytest.mark.parametrize("n", [2393, 2395, 3001])
def test_large_readbacks_equal_small_ones(n):
    """Reads on both sides of where the readback's lanes start (4 MB: 2,394
    slots' bodies, 2,341 slots' rings of 8), with a last chunk that is not
    full: the whole read equals reads of 250 slots, also from two threads at
    once."""
    from concurrent.futures import ThreadPoolExecutor

    from kraken_3_gpu_b200 import batch, workloads
    w = workloads.uneven(n=n, n_maps=2, seed=4, h_min=3, h_max=9)
    eng = batch.BatchEngine(w.maps, w.n, obs_ring=8)
    workloads.spawn_all(eng, w)
    eng.run(9)
    parts = [eng.read_state(i, min(250, n - i)) for i in range(0, n, 250)]
    obs = np.concatenate([eng.read_obs(i, min(250, n - i)) for i in range(0, n, 250)])
    with ThreadPoolExecutor(2) as pool:
        whole = list(pool.map(lambda _: (eng.read_state(), eng.read_obs()), range(2)))
    for st, ob in whole:
        for f in ("px", "py", "vx", "vy", "ang", "av", "grips", "steps"):
            assert np.array_equal(st[f], np.concatenate([p[f] for p in parts])), f
        assert np.array_equal(ob, obs)
    eng.close()
