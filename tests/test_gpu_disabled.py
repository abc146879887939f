"""Drop-in worlds whose broken constraints hold values that no live one could:
the step must leave them out as the f32 oracle does."""
import ctypes as C

import numpy as np
import pytest

from kraken_3_gpu_b200 import _native
from oracle import binding as ob

pytestmark = pytest.mark.gpu

_F32P, _U32P = C.POINTER(C.c_float), C.POINTER(C.c_uint32)
RECTS = np.array([[0, 0, 400, 14], [0, 286, 400, 14], [0, 0, 14, 300], [386, 0, 14, 300]], float)


@pytest.mark.parametrize("lever", [7.0, 1e25, np.inf, np.nan])
@pytest.mark.parametrize("angle", [0.3, 70.0, 1e17, -np.inf])
def test_broken_constraints_touch_nothing(lever, angle):
    """Pairs of bodies joined by a broken pin, a broken grip or a broken angle
    constraint each, one body of each pair at `angle`, the broken records'
    levers, targets and compliances `lever`; a live pin on the other body of
    some pairs.  Every body equals the oracle's, whose step skips what is
    broken, in every field that the oracle leaves finite or not."""
    o = ob.World()
    o.set_rects(RECTS)
    r = np.random.default_rng(2)
    for k in range(24):
        a = o.add_body(r.uniform(60, 340), r.uniform(60, 240), angle if k % 2 else 0.4, 3.0, 90.0)
        b = o.add_body(r.uniform(60, 340), r.uniform(60, 240), 0.2, 2.0, 70.0)
        if k % 3 == 0:  # a live pin of another pair's kind: the group still solves
            c = o.add_constraint(0, b, -1, 5, 1, r.uniform(100, 300), r.uniform(100, 200), 0.0)
        c = o.add_constraint(k % 3, a, b if k % 4 else -1, lever, 1.0, 2.0, lever, lever)
        c.rest, c.target = lever, lever
        c.minAngle, c.maxAngle, c.breakForce = -1.0, 1.0, 100.0
        c.broken = True
    o.set_list(np.arange(o.nC))
    o.f32ify()
    o.round_state()
    n = o.n
    bodies = np.zeros((n, 12), np.float32)
    for i, f in enumerate(("px", "py", "ppx", "ppy", "vx", "vy", "ang", "angP", "av", "im", "ii")):
        bodies[:, i] = o.arr(f)
    cons = np.zeros((o.nC, 20), np.float32)
    cu = cons.view(np.uint32)
    for k, c in enumerate(o.constraints):
        cu[k, 0], cu[k, 1], cu[k, 2] = c.a, c.b & 0xFFFFFFFF, c.type
        cons[k, 4:13] = (c.lax, c.lay, c.lbx, c.lby, c.compliance, c.rest, c.target, c.minAngle, c.maxAngle)
        cons[k, 16] = c.breakForce
        cu[k, 17] = c.broken
    L, h = _native.lib(), C.c_void_p()
    p = _native.SolverParams(1 / 120, 2, 4, 3.0, 3.0, 360.0, 18.0)
    r32 = RECTS.astype(np.float32)
    _native.check(L.kr_create(C.byref(p), n, o.nC, r32.ctypes.data_as(_F32P), len(r32), None, 0, None, C.byref(h)))
    try:
        cp = cons.ctypes.data_as(_U32P)
        _native.check(L.kr_upload(h, bodies.ctypes.data_as(_F32P), cp, None, None), h)
        for s in range(2):
            _native.check(L.kr_step(h, 1), h)
            _native.check(L.kr_download(h, bodies.ctypes.data_as(_F32P), cp), h)
            o.step32()
            for c, f in ((0, "px"), (1, "py"), (2, "ppx"), (3, "ppy"), (4, "vx"), (5, "vy"), (7, "angP")):
                assert np.array_equal(bodies[:, c], o.arr(f).astype(np.float32), equal_nan=True), (s, f)
    finally:
        L.kr_destroy(h)
