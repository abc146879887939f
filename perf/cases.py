"""The work a user has this framework do, as timed cases.

Four entry points: the gpuworld drop-in (``kr_upload`` / ``kr_upload_controls``
/ ``kr_step`` / ``kr_download``), the allocation-free step (``kr_step_noalloc``),
the batched engine (``kraken_3_gpu_b200.batch.BatchEngine``) under each of its
controllers, and the rollout server (``kraken_3_gpu_b200.serve.Server``).
Sizes are those of the configurations, tests and benchmark of this repository,
and the ranges between them.

A case's ``kind`` says which path it takes; every pass starts from the same
state (an upload, a restored snapshot, fresh requests), so it can be repeated.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from kraken_3_gpu_b200 import _native, batch, core, gpuworld, kraken, serve, workloads

_F32P = C.POINTER(C.c_float)
_U32P = C.POINTER(C.c_uint32)

DT = 1 / 120
SUBSTEPS, ITERATIONS = 2, 4


def listed():
    return [
        # one creature on screen: the page's loop of a second's 60 env steps,
        # controls up and state down around every step (latency)
        {"name": "dropin_frames_1", "kind": "dropin", "creatures": 1, "arms": 6, "segs": 7, "frames": 60,
         "per_frame": 1},
        # a small population of the largest body, stepped in the same loop
        {"name": "dropin_frames_64", "kind": "dropin", "creatures": 64, "arms": 8, "segs": 9, "frames": 12,
         "per_frame": 1},
        # a population of the default body rolled out between two readbacks
        {"name": "dropin_rollout_1024", "kind": "dropin", "creatures": 1024, "arms": 6, "segs": 7, "frames": 2,
         "per_frame": 100},
        # an embedding that owns its device memory: a step on its own buffers
        {"name": "noalloc_40", "kind": "noalloc", "creatures": 40, "arms": 6, "segs": 7, "steps": 4},
        # an external controller that reads the proprioception of every step
        {"name": "external_200", "kind": "external", "creatures": 200, "arms": 5, "segs": 6, "steps": 1},
        # a handful of creatures evaluated for two seconds (latency)
        {"name": "stream_12", "kind": "stream", "creatures": 12, "arms": 6, "segs": 7, "steps": 120, "maps": 1,
         "uneven": False},
        # an ES generation of the default body on one map
        {"name": "stream_1024", "kind": "stream", "creatures": 1024, "arms": 6, "segs": 7, "steps": 400, "maps": 1,
         "uneven": False},
        # the headline: uneven bodies, maps and horizons 200..2000, regrouped
        # in time slices
        {"name": "uneven_16384", "kind": "stream", "creatures": 16384, "arms": 0, "segs": 0, "steps": 2000,
         "maps": 64, "uneven": True},
        # creatures under the fused policy, weights of their own
        {"name": "policy_3000", "kind": "policy", "creatures": 3000, "arms": 0, "segs": 0, "steps": 300, "maps": 16,
         "uneven": True},
        # creatures under the reference trainer's net with its senses
        {"name": "net_2500", "kind": "net", "creatures": 2500, "arms": 0, "segs": 0, "steps": 240, "maps": 16,
         "uneven": True},
        # the memory-bound form: every creature keeps an observation ring
        {"name": "ring_6000", "kind": "ring", "creatures": 6000, "arms": 0, "segs": 0, "steps": 320, "maps": 32,
         "uneven": True},
        # a rollout server's ES requests: mirrored populations around theta
        {"name": "server_es_24", "kind": "server", "requests": 24, "population": 96, "horizon": 500, "maps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "noalloc", "external", "stream", "stream", "policy", "net", "ring", "server"])
    arms, segs = rng.randint(4, 8), rng.randint(5, 9)
    if kind == "dropin":
        n = _log(rng, 1, 1024)
        if rng.random() < 0.5:
            return {"kind": kind, "creatures": n, "arms": arms, "segs": segs, "frames": rng.randint(6, 40),
                    "per_frame": 1}
        return {"kind": kind, "creatures": n, "arms": arms, "segs": segs, "frames": rng.randint(1, 3),
                "per_frame": rng.randint(10, 80)}
    if kind == "noalloc":
        most = min(2048 // (1 + arms * segs), 4096 // (2 * arms * segs + arms), 4096 // (8 + 2 * arms * segs))
        return {"kind": kind, "creatures": _log(rng, 1, most), "arms": arms, "segs": segs, "steps": rng.randint(1, 10)}
    if kind == "external":
        return {"kind": kind, "creatures": _log(rng, 1, 2000), "arms": arms, "segs": segs, "steps": rng.randint(1, 4)}
    if kind == "server":
        return {"kind": kind, "requests": rng.randint(3, 40), "population": 2 * rng.randint(4, 128),
                "horizon": rng.randint(100, 900), "maps": rng.randint(1, 16)}
    if rng.random() < 0.3:
        return {"kind": kind, "creatures": _log(rng, 1, 3000), "arms": arms, "segs": segs,
                "steps": _log(rng, 20, 600), "maps": 1, "uneven": False}
    return {"kind": kind, "creatures": _log(rng, 100, 9000), "arms": 0, "segs": 0, "steps": _log(rng, 100, 900),
            "maps": rng.randint(1, 64), "uneven": True}


# --- inputs -----------------------------------------------------------------

def _map(density, seed):
    return workloads.make_map(workloads.WIDTH, workloads.HEIGHT, seed=seed, density=density)


def _poses(case, seed):
    """Spawn poses of a one-shape population on one map: findSpawn's points
    with jitter, any heading."""
    r = np.random.default_rng(seed)
    m = _map(0.48, 1 + seed % 97)
    rnd = workloads.mulberry32(int(r.integers(1 << 32)))
    n = case["creatures"]
    pts = [workloads.find_spawn(m, kraken.arm_reach(case["segs"]) + 20, rnd) for _ in range(min(n, 16))]
    k = r.integers(len(pts), size=n)
    xy = np.array([[p["x"], p["y"]] for p in pts])[k] + r.uniform(-20, 20, (n, 2))
    return m, xy, r.uniform(0, 2 * math.pi, n), r


def _world(case, seed):
    """A world of one body shape as the drop-in's blocks: bodies (nB, 12) f32,
    constraints (nC, 20) words in solve-list order, collision points, ranges,
    rects, and the motors' control sets (one per 6 env steps)."""
    m, xy, ang, r = _poses(case, seed)
    n, A, S = case["creatures"], case["arms"], case["segs"]
    sim = core.create_sim(seed=1, poses=[(0.0, 0.0, 0.0)], arms=A, segsPerArm=S)
    w = sim["world"]
    nb, nc, npt = w.n, len(w.constraints), len(w.collPts)
    # spawnKraken's pose at the origin, turned and moved
    c, s = np.cos(ang)[:, None], np.sin(ang)[:, None]
    px = xy[:, :1] + c * w.px[:nb] - s * w.py[:nb]
    py = xy[:, 1:] + s * w.px[:nb] + c * w.py[:nb]
    th = ang[:, None] + w.ang[:nb]
    bodies = np.zeros((n, nb, 12), np.float32)
    bodies[..., 0], bodies[..., 1], bodies[..., 2], bodies[..., 3] = px, py, px, py
    bodies[..., 6], bodies[..., 7] = th, th
    bodies[..., 9], bodies[..., 10] = w.im[:nb], w.ii[:nb]
    one = np.zeros((nc, 20), np.float32)
    ou = one.view(np.uint32)
    color = np.zeros(nc, np.int64)
    for k, q in enumerate(w.constraints):
        ou[k, 0], ou[k, 1], ou[k, 2] = q.a, q.b if q.b >= 0 else 0xFFFFFFFF, q.type
        one[k, 4:13] = (q.lax, q.lay, q.lbx, q.lby, kraken.tone_to_compliance(0.5) if q.type == 1 else 0.0, q.rest,
                        0.0, q.minAngle, q.maxAngle)
        ou[k, 17] = 1 if q.type == 2 else 0
        color[k] = q.color
    cons = np.tile(one, (n, 1, 1))
    cu = cons.view(np.uint32)
    off = (np.arange(n, dtype=np.uint32) * nb)[:, None]
    cu[..., 0] += off
    cu[..., 1] = np.where(cu[..., 1] == 0xFFFFFFFF, cu[..., 1], cu[..., 1] + off)
    motors = np.nonzero(ou[:, 2] == 1)[0]
    grips = np.nonzero(ou[:, 2] == 2)[0]
    # every cup whose adhesion exceeds the attach threshold holds from the start
    adh = r.uniform(0, 1, (n, len(grips)))
    tips = ou[grips, 0].astype(np.int64)
    held = adh > 0.08
    tip = bodies[:, tips].astype(np.float64)
    cons[:, grips, 6] = np.where(held, tip[..., 0] + 6.75 * np.cos(tip[..., 6]), cons[:, grips, 6])
    cons[:, grips, 7] = np.where(held, tip[..., 1] + 6.75 * np.sin(tip[..., 6]), cons[:, grips, 7])
    cons[:, grips, 16] = np.where(held, 40 + 860 * adh, 0)
    cu[:, grips, 17] = ~held
    order = np.argsort(np.broadcast_to(color, (n, nc)).ravel(), kind="stable")
    cons = np.ascontiguousarray(cons.reshape(-1, 20)[order])
    place = np.empty(n * nc, np.int64)
    place[order] = np.arange(n * nc)
    mot = place.reshape(n, nc)[:, motors]
    lim = np.abs(one[motors, 11])
    grouped = gpuworld.groupCollPoints(w.collPts, nb)
    pts = np.zeros((n, npt, 4), np.float32)
    for o, i in enumerate(grouped["order"]):
        q = w.collPts[int(i)]
        pts[:, o, 1:] = (q.lx, q.ly, q.r)
        pts.view(np.uint32)[:, o, 0] = q.body + off[:, 0]
    cnt = np.tile(grouped["range"][nb:], n).astype(np.uint32)
    rng = np.concatenate([np.concatenate([[0], np.cumsum(cnt)[:-1]]).astype(np.uint32), cnt]).astype(np.uint32)
    rects = np.array([[q["x"], q["y"], q["w"], q["h"]] for q in m["rects"]], np.float32)
    sets = [np.clip(r.uniform(-1, 1, (n, len(motors))), -lim, lim).astype(np.float32) for _ in range(10)]
    return {"n": n, "nb": nb, "nc": nc, "bodies": bodies.reshape(-1, 12), "cons": cons, "pts": pts.reshape(-1, 4),
            "range": rng, "rects": rects, "mot": mot, "sets": sets, "place": place.reshape(n, nc)}


def _params():
    return _native.SolverParams(DT, SUBSTEPS, ITERATIONS, 3.0, 3.0, 360.0, 18.0)


def _workload(case, seed):
    if case.get("uneven"):
        return workloads.uneven(n=case["creatures"], n_maps=case["maps"], seed=2 + seed % 100003,
                                h_min=max(1, case["steps"] // 10), h_max=case["steps"])
    m, xy, ang, r = _poses(case, seed)
    n = case["creatures"]
    one = np.ones(n, np.int32)
    lights = [np.array(workloads.light_array(m), np.float64).reshape(-1, 6)]
    return workloads.Workload("one shape", [workloads._rects(m)], case["arms"] * one, case["segs"] * one, 0 * one,
                              xy[:, 0], xy[:, 1], ang, case["steps"] * one,
                              r.integers(1 << 32, size=n, dtype=np.uint64).astype(np.uint32), lights)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        w = _world(case, seed)
        L = _native.lib()
        h = C.c_void_p()
        p = _params()
        _native.check(L.kr_create(C.byref(p), len(w["bodies"]), len(w["cons"]), w["rects"].ctypes.data_as(_F32P),
                                  len(w["rects"]), w["pts"].ctypes.data_as(_U32P), len(w["pts"]),
                                  w["range"].ctypes.data_as(_U32P), C.byref(h)))
        return _DropIn(case, w, h)
    if kind == "noalloc":
        w = _world(case, seed)
        w["cons"][w["mot"], 10] = w["sets"][0]
        dev = {k: torch.from_numpy(np.ascontiguousarray(w[k]).view(np.int32)).cuda()
               for k in ("bodies", "cons", "pts", "range", "rects")}
        L = _native.lib()
        L.kr_step_noalloc.restype = C.c_int
        L.kr_step_noalloc.argtypes = [C.POINTER(_native.SolverParams), C.c_uint32, C.c_uint32, C.c_void_p, C.c_void_p,
                                      C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_uint32, C.c_void_p,
                                      C.c_int32, C.c_void_p]
        return {"case": case, "w": w, "dev": dev, "bodies": torch.empty_like(dev["bodies"]),
                "cons": torch.empty_like(dev["cons"]), "params": _params(),
                "forces": torch.zeros((len(w["bodies"]), 4), device="cuda")}
    if kind == "server":
        return _Requests(case, seed)
    w = _workload(case, seed)
    r = np.random.default_rng(seed + 1)
    control = {"external": "buffer", "ring": "stream"}.get(kind, kind)
    eng = batch.BatchEngine(w.maps, w.n, obs_ring={"ring": 128, "external": 1}.get(kind, 0), control=control,
                            lights=w.lights if control == "net" else None)
    workloads.spawn_all(eng, w)
    state = {"case": case, "eng": eng, "w": w}
    if kind == "external":
        c = np.zeros((w.n, batch.CTRL_STRIDE), np.float32)
        A, S = case["arms"], case["segs"]
        c[:, :A * S] = r.uniform(-1, 1, (w.n, A * S))
        c[:, A * S:A * S + A] = r.uniform(0, 1, (w.n, A))
        state["controls"] = c
    elif kind == "policy":
        n = max(batch.policy_params(int(a), int(s)) for a, s in zip(w.arms, w.segs))
        g = torch.Generator(device="cuda").manual_seed(seed)
        eng.set_policy((torch.randn((w.n, n), generator=g, device="cuda") * 0.1).cpu().numpy(), np.arange(w.n))
    elif kind == "net":
        n = batch.net_param_count(int(w.arms.max()))
        g = torch.Generator(device="cuda").manual_seed(seed)
        eng.set_net((torch.randn((w.n, n), generator=g, device="cuda") * 0.3).cpu().numpy(), np.arange(w.n))
    if kind in ("stream", "policy", "net", "ring") and case["uneven"]:
        eng.set_slice(50.0)
    eng.snapshot()
    return state


class _DropIn:
    """A world behind a drop-in handle, with the host blocks its loop reuses."""

    def __init__(self, case, w, h):
        self.case, self.w, self.h = case, w, h
        self.bodies, self.cons = w["bodies"].copy(), w["cons"].copy()

    def __del__(self):
        if self.h:
            _native.lib().kr_destroy(self.h)
            self.h = None


class _Requests:
    """A server and the requests of one pass."""

    def __init__(self, case, seed):
        r = np.random.default_rng(seed)
        size = np.random.default_rng(case["requests"] * 1000003 + case["population"] * 1009 + case["horizon"])
        self.case = case
        maps = [_map(float(r.uniform(0.1, 0.4)), int(r.integers(1 << 30))) for _ in range(case["maps"])]
        self.srv = serve.Server([workloads._rects(m) for m in maps], hbm_budget=4 << 30, max_slots=4096, slice_ms=50.0)
        self.reqs = []
        for _ in range(case["requests"]):
            A, S, k = int(size.integers(4, 9)), int(size.integers(5, 10)), int(r.integers(case["maps"]))
            sp = workloads.find_spawn(maps[k], kraken.arm_reach(S) + 20, workloads.mulberry32(int(r.integers(1 << 32))))
            pop = 2 * int(size.integers(max(1, case["population"] // 4), case["population"] // 2 + 1))
            self.reqs.append(dict(population=pop, horizon=int(size.integers(case["horizon"] // 3, case["horizon"] + 1)),
                                  arms=A, segs=S, map_id=k, x=sp["x"], y=sp["y"], angle=float(r.uniform(0, 6.28)),
                                  theta=r.normal(0, 0.1, batch.policy_params(A, S)).astype(np.float32), sigma=0.02,
                                  seed=int(r.integers(1 << 40))))


# --- one pass ---------------------------------------------------------------

def run(state):
    if isinstance(state, _DropIn):
        return _run_dropin(state)
    if isinstance(state, _Requests):
        s = state.srv
        ids = [s.submit(**q) for q in state.reqs]
        s.drain()
        return list(s.results_many(ids, [q["population"] for q in state.reqs], release=True)[0].T)
    if state["case"]["kind"] == "noalloc":
        w, d = state["w"], state["dev"]
        state["bodies"].copy_(d["bodies"])
        state["cons"].copy_(d["cons"])
        rc = _native.lib().kr_step_noalloc(
            C.byref(state["params"]), len(w["bodies"]), len(w["cons"]), state["bodies"].data_ptr(),
            state["cons"].data_ptr(), state["forces"].data_ptr(), d["rects"].data_ptr(), len(w["rects"]),
            d["pts"].data_ptr(), len(w["pts"]), d["range"].data_ptr(), state["case"]["steps"],
            torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError(f"kr_step_noalloc: status {rc}")
        c = state["cons"]
        return {"bodies": state["bodies"].view(torch.float32), "lambda": c[:, 13:16].view(torch.float32),
                "broken": c[:, 17]}
    eng, case = state["eng"], state["case"]
    eng.restore()
    out = {}
    if case["kind"] == "external":
        for s in range(case["steps"]):
            eng.set_controls(state["controls"])
            eng.run(1)
            out["obs%d" % s] = eng.read_obs()[:, :, :6 * case["arms"] + 6]
    else:
        eng.run(case["steps"])
        if case["kind"] == "ring":
            out["obs"] = eng.read_obs()
            out["flags"] = out["obs"][:, :, -1].view(np.int32)
            out["obs"] = out["obs"][:, :, :-1]
    st = eng.read_state()
    out.update({f: st[f] for f in ("px", "py", "ang", "vx", "vy", "av", "steps")})
    out["held"] = (st["grips"][..., 3] == 0).astype(np.int32)
    out["metrics"] = list(eng.read_metrics().T)
    return out


def _run_dropin(s):
    L, h, case, w = _native.lib(), s.h, s.case, s.w
    bp, cp = s.bodies.ctypes.data_as(_F32P), s.cons.ctypes.data_as(_U32P)
    _native.check(L.kr_upload(h, w["bodies"].ctypes.data_as(_F32P), w["cons"].ctypes.data_as(_U32P), None, None), h)
    s.cons[:] = w["cons"]
    for f in range(case["frames"]):
        if case["per_frame"] > 1 or f % 6 == 0:
            s.cons[w["mot"], 10] = w["sets"][(f if case["per_frame"] > 1 else f // 6) % len(w["sets"])]
        _native.check(L.kr_upload_controls(h, cp), h)
        _native.check(L.kr_step(h, case["per_frame"]), h)
        _native.check(L.kr_download(h, bp, cp), h)
    return {"bodies": s.bodies.copy(), "lambda": s.cons[:, 13:16].copy(),
            "broken": s.cons.view(np.int32)[:, 17].copy()}


def _creature_steps(case):
    """(creature-steps, mean bodies per creature, creatures) of a pass."""
    if case["kind"] == "server":
        n = case["requests"] * case["population"] * 0.75
        return n * case["horizon"] * 2 / 3, 43.0, n
    n = case["creatures"]
    if case["kind"] == "dropin":
        return n * case["frames"] * case["per_frame"], 1 + case["arms"] * case["segs"], n
    if case["kind"] in ("noalloc", "external") or not case["uneven"]:
        return n * case["steps"], 1 + case["arms"] * case["segs"], n
    return n * case["steps"] * 0.55, 43.0, n


def work(case):
    """Per joint and iteration a pin (two sine / cosine pairs, a 2 x 2 solve)
    and a muscle with its limit, per body and iteration one test against the
    walls, per body and substep the integration and the velocity update."""
    steps, nb, n = _creature_steps(case)
    per_step = SUBSTEPS * (ITERATIONS * ((nb - 1) * 230 + nb * 10) + nb * 60)
    extra = {"policy": 2 * 64 * (42 + 49), "server": 2 * 64 * (42 + 49), "net": 2 * (24 * (105 + 24 + 20))}
    flops = steps * (per_step + extra.get(case["kind"], 0))
    bytes_ = n * nb * 48 * 2
    if case["kind"] == "dropin":
        bytes_ = n * nb * 48 * (1 + case["frames"]) + n * (nb - 1) * 2 * 80 * (1 + 2 * case["frames"])
    if case["kind"] in ("policy", "server", "net"):
        bytes_ += n * 4 * (64 * (42 + 49) if case["kind"] != "net" else 24 * 149)
    if case["kind"] == "ring":
        bytes_ += n * 128 * 56 * 4
    return {"bytes": float(bytes_), "flops": float(flops)}


# --- the same in 64 bits ----------------------------------------------------

def exact(case, seed):
    """The step's equations in numpy f64 from the same f32 inputs, where that
    takes seconds: the drop-in, the allocation-free step, one step of the
    external controller and small stream-controlled populations."""
    kind = case["kind"]
    if kind == "external" and case["steps"] == 1 or kind == "stream" and not case["uneven"]:
        steps = case["steps"]
    elif kind == "noalloc":
        steps = case["steps"]
    elif kind == "dropin":
        steps = case["frames"] * case["per_frame"]
    else:
        return None
    if case["creatures"] * steps > 2500 or steps > 200:
        return None
    if kind in ("external", "stream"):
        return _exact_engine(case, seed)
    w = _world(case, seed)
    x = _Solver64(w)
    for s in range(steps):
        f = s // case["per_frame"] if kind == "dropin" else 0
        at = 0 if kind == "noalloc" else f if case["per_frame"] > 1 else f // 6
        x.target(w["sets"][at % len(w["sets"])])
        x.step()
    bodies = w["bodies"].astype(np.float64).reshape(w["n"], w["nb"], 12)
    for c, v in zip((0, 1, 2, 3, 4, 5, 6, 7, 8), (x.px, x.py, x.qx, x.qy, x.vx, x.vy, x.an, x.qa, x.av)):
        bodies[..., c] = v
    lam = np.zeros((w["n"] * w["nc"], 3))
    lam[w["place"]] = np.stack([x.lx, x.ly, x.la], -1)
    return {"bodies": bodies.reshape(-1, 12), "lambda": lam, "broken": None}


def _draws(state, count):
    """The next `count` draws of every mulberry32 stream, and its state after them."""
    out = []
    for _ in range(count):
        state = state + np.uint32(0x6D2B79F5)
        t = (state ^ (state >> np.uint32(15))) * (state | np.uint32(1))
        t ^= t + (t ^ (t >> np.uint32(7))) * (t | np.uint32(61))
        out.append((t ^ (t >> np.uint32(14))) / 4294967296.0)
    return np.stack(out, -1), state


def _exact_engine(case, seed):
    """From the spawn pose, per step: the controls (given, or the stream's
    draws every 6 steps), the suction-cup reflex, the step."""
    w = _workload(dict(case, uneven=False), seed)
    A, S, n = case["arms"], case["segs"], case["creatures"]
    world = _world(case, seed)
    b = world["bodies"].reshape(n, world["nb"], 12)
    # spawnKraken's chain in f64, rounded once
    px, py, th = np.zeros((n, world["nb"])), np.zeros((n, world["nb"])), np.zeros((n, world["nb"]))
    px[:, 0], py[:, 0], th[:, 0] = w.x, w.y, w.angle
    k = 1
    for a in range(A):
        t = w.angle + a / A * math.pi * 2
        jx, jy = w.x + np.cos(t) * 24, w.y + np.sin(t) * 24
        for _ in range(S):
            px[:, k], py[:, k], th[:, k] = jx + np.cos(t) * 6.75, jy + np.sin(t) * 6.75, t
            jx, jy = jx + np.cos(t) * 13.5, jy + np.sin(t) * 13.5
            t = t + 0.28
            k += 1
    b[..., 0], b[..., 1], b[..., 6] = px, py, th
    x = _Solver64(world)
    g = np.nonzero(x.kind == 2)[0]
    g = g[np.argsort(x.a[g])]  # by arm
    tips = x.a[g]
    x.broken[:, g] = True
    # motors in solve-list order: the joint of an arm's segment is its motor
    seg = x.b[x.mot] - 1
    lim = np.where(seg % S == 0, math.pi * 0.62, math.pi * 0.42)
    if case["kind"] == "external":
        r = np.random.default_rng(seed + 1)
        targets = r.uniform(-1, 1, (n, A * S)).astype(np.float32).astype(np.float64)
        adh = r.uniform(0, 1, (n, A)).astype(np.float32).astype(np.float64)
    rng, cd = w.seed, np.zeros((n, A))
    for s in range(case["steps"]):
        if case["kind"] == "stream" and s % 6 == 0:
            d, rng = _draws(rng, A * (S + 1))
            d = d.reshape(n, A, S + 1)
            targets = (d[..., :S] * 2 - 1).reshape(n, -1).astype(np.float32).astype(np.float64)
            adh = d[..., S].astype(np.float32).astype(np.float64)
        x.tgt[:, x.mot] = np.clip(targets[:, seg], -lim, lim)
        cd = np.where(cd > 0, cd - DT * SUBSTEPS, cd)
        free = x.broken[:, g]
        want = free & (adh > 0.08) & (cd <= 0)
        hold = want & (np.hypot(x.vx[:, tips], x.vy[:, tips]) < 150)
        cd = np.where(want & ~hold, 0.05, cd)
        x.lbx[:, g] = np.where(hold, x.px[:, tips] + 6.75 * np.cos(x.an[:, tips]), x.lbx[:, g])
        x.lby[:, g] = np.where(hold, x.py[:, tips] + 6.75 * np.sin(x.an[:, tips]), x.lby[:, g])
        x.brk[:, g] = np.where(hold | ~free, 40 + 860 * adh, x.brk[:, g])
        x.broken[:, g] = np.where(free, ~hold, adh < 0.04)
        x.step()
    out = {f: np.zeros((n, batch.MAX_BODIES)) for f in ("px", "py", "ang", "vx", "vy", "av")}
    for f, v in zip(out, (x.px, x.py, x.an, x.vx, x.vy, x.av)):
        out[f][:, :world["nb"]] = v
    return {**out, "obs0": None, "steps": None, "held": None, "metrics": None}


def _delta(a, b):
    d = np.fmod(a - b, 2 * math.pi)
    return np.where(d > math.pi, d - 2 * math.pi, np.where(d < -math.pi, d + 2 * math.pi, d))


class _Solver64:
    """The XPBD step of a one-shape population, every array (creature, body)
    or (creature, constraint), one colour class of constraints at a time."""

    def __init__(self, w):
        n, nb = w["n"], w["nb"]
        b = w["bodies"].astype(np.float64).reshape(n, nb, 12)
        self.px, self.py, self.vx, self.vy, self.an, self.av = (b[..., c].copy() for c in (0, 1, 4, 5, 6, 8))
        self.im, self.ii = b[0, :, 9], b[0, :, 10]
        c = w["cons"][w["place"]]
        u = c.view(np.uint32)
        c = c.astype(np.float64)
        self.a = u[0, :, 0].astype(np.int64)
        self.b = np.where(u[0, :, 1] == 0xFFFFFFFF, -1, u[0, :, 1].astype(np.int64))
        self.kind = u[0, :, 2].astype(np.int64)
        self.lax, self.lay, self.lbx, self.lby, self.comp, self.rest, self.tgt, self.mn, self.mx = (
            c[..., k].copy() for k in range(4, 13))
        self.brk, self.broken = c[..., 16].copy(), u[..., 17] != 0
        # the list order of one creature, split into body-disjoint runs
        runs, used = [[]], set()
        for k in range(w["nc"]):
            bs = {int(self.a[k]), int(self.b[k])} - {-1}
            if bs & used or (runs[-1] and (self.kind[runs[-1][0]] == 1) != (self.kind[k] == 1)):
                runs.append([])
                used = set()
            runs[-1].append(k)
            used |= bs
        self.runs = [np.array(q) for q in runs]
        self.mot = np.nonzero(self.kind == 1)[0]
        p = w["pts"].reshape(n, -1, 4)[0]
        body = p.view(np.uint32)[:, 0].astype(np.int64)
        p = p.astype(np.float64)
        self.pts = [[] for _ in range(8)]
        seen = {}
        for k in range(len(p)):
            j = seen.get(int(body[k]), 0)
            seen[int(body[k])] = j + 1
            self.pts[j].append((int(body[k]), *p[k, 1:]))
        self.pts = [np.array(q).T for q in self.pts if q]
        self.rects = w["rects"].astype(np.float64)

    def target(self, t):
        self.tgt[:, self.mot] = t

    def step(self):
        for _ in range(SUBSTEPS):
            self.substep()
        g = np.nonzero(self.kind == 2)[0]
        broke = ~self.broken[:, g] & (np.hypot(self.lx[:, g], self.ly[:, g]) / DT > self.brk[:, g])
        self.broken[:, g] |= broke
        self.lx[:, g] = np.where(broke, 0, self.lx[:, g])
        self.ly[:, g] = np.where(broke, 0, self.ly[:, g])

    def substep(self):
        damp = math.exp(-3.0 * DT)
        self.lx, self.ly, self.la = (np.zeros_like(self.lax) for _ in range(3))
        vx, vy, av = self.vx * damp, self.vy * damp, np.clip(self.av * damp, -18, 18)
        sp = np.hypot(vx, vy)
        k = np.where(sp > 360, 360 / np.maximum(sp, 1e-9), 1)
        self.qx, self.qy, self.qa = self.px + DT * vx * k, self.py + DT * vy * k, self.an + DT * av
        for _ in range(ITERATIONS):
            for r in self.runs:
                if self.kind[r[0]] == 1:
                    self.angles(r)
                else:
                    self.pins(r)
            self.walls()
        vx, vy = (self.qx - self.px) / DT, (self.qy - self.py) / DT
        sp = np.hypot(vx, vy)
        k = np.where(sp > 360, 360 / np.maximum(sp, 1e-9), 1)
        self.vx, self.vy = vx * k, vy * k
        self.av = np.clip(_delta(self.qa, self.an) / DT, -18, 18)
        self.qa = np.where(np.abs(self.qa) > 50, _delta(self.qa, 0.0), self.qa)
        self.px, self.py, self.an = self.qx.copy(), self.qy.copy(), self.qa.copy()

    def pins(self, r):
        a, b = self.a[r], self.b[r]
        has = b >= 0
        bb = np.where(has, b, 0)
        ca, sa, cb, sb = np.cos(self.qa[:, a]), np.sin(self.qa[:, a]), np.cos(self.qa[:, bb]), np.sin(self.qa[:, bb])
        lax, lay, lbx, lby = (v[:, r] for v in (self.lax, self.lay, self.lbx, self.lby))
        rax, ray = lax * ca - lay * sa, lax * sa + lay * ca
        rbx, rby = np.where(has, lbx * cb - lby * sb, 0), np.where(has, lbx * sb + lby * cb, 0)
        cx = self.qx[:, a] + rax - np.where(has, self.qx[:, bb] + rbx, lbx)
        cy = self.qy[:, a] + ray - np.where(has, self.qy[:, bb] + rby, lby)
        wa, ia = self.im[a], self.ii[a]
        wb, ib = np.where(has, self.im[bb], 0), np.where(has, self.ii[bb], 0)
        k00 = wa + wb + ia * ray * ray + ib * rby * rby
        k01 = -ia * ray * rax - ib * rby * rbx
        k11 = wa + wb + ia * rax * rax + ib * rbx * rbx
        det = k00 * k11 - k01 * k01
        on = ~self.broken[:, r] & (cx * cx + cy * cy >= 4e-6) & (np.abs(det) >= 1e-12)
        det = np.where(on, det, 1)
        dx = np.where(on, -(k11 * cx - k01 * cy) / det, 0)
        dy = np.where(on, -(k00 * cy - k01 * cx) / det, 0)
        self.lx[:, r] += dx
        self.ly[:, r] += dy
        self.qx[:, a] += wa * dx
        self.qy[:, a] += wa * dy
        self.qa[:, a] += ia * (rax * dy - ray * dx)
        b = b[has]
        self.qx[:, b] -= (wb * dx)[:, has]
        self.qy[:, b] -= (wb * dy)[:, has]
        self.qa[:, b] -= (ib * (rbx * dy - rby * dx))[:, has]

    def angles(self, r):
        a, b = self.a[r], self.b[r]
        wa, wb = self.ii[a], self.ii[b]
        c = _delta(_delta(_delta(self.qa[:, b], self.qa[:, a]), self.rest[:, r]), self.tgt[:, r])
        al = self.comp[:, r] / (DT * DT)
        dl = np.where(np.abs(c) >= 2e-4, -(c + al * self.la[:, r]) / (wa + wb + al), 0)
        self.la[:, r] += dl
        self.qa[:, b] += wb * dl
        self.qa[:, a] -= wa * dl
        d = _delta(_delta(self.qa[:, b], self.qa[:, a]), self.rest[:, r])
        over = np.where(d > self.mx[:, r], d - self.mx[:, r], np.where(d < self.mn[:, r], d - self.mn[:, r], 0))
        dl = np.where(np.abs(over) >= 2e-4, -over / (wa + wb), 0)
        self.qa[:, b] += wb * dl
        self.qa[:, a] -= wa * dl

    def walls(self):
        c, s = np.cos(self.qa), np.sin(self.qa)
        for q in self.pts:
            j = q[0].astype(np.int64)
            x = self.qx[:, j] + q[1] * c[:, j] - q[2] * s[:, j]
            y = self.qy[:, j] + q[1] * s[:, j] + q[2] * c[:, j]
            best, nx, ny = np.full(x.shape, np.inf), np.zeros(x.shape), np.zeros(x.shape)
            for rx, ry, rw, rh in self.rects:
                dx, dy = x - np.clip(x, rx, rx + rw), y - np.clip(y, ry, ry + rh)
                d2 = dx * dx + dy * dy
                out = (d2 > 1e-12) & (d2 < best * best)
                d = np.sqrt(np.where(d2 > 0, d2, 1))
                nx, ny, best = np.where(out, dx / d, nx), np.where(out, dy / d, ny), np.where(out, d, best)
                m = np.stack([x - rx, rx + rw - x, y - ry, ry + rh - y])
                k = np.argmin(m, 0)
                m = np.min(m, 0)
                inn = (d2 <= 1e-12) & (-m < best)
                nx = np.where(inn, np.array([-1.0, 1, 0, 0])[k], nx)
                ny = np.where(inn, np.array([0.0, 0, -1, 1])[k], ny)
                best = np.where(inn, -m, best)
            pen = q[3] - best
            hit = pen > 2e-3
            self.qx[:, j] += np.where(hit, nx * pen, 0)
            self.qy[:, j] += np.where(hit, ny * pen, 0)
