"""The batched engine where the near sets are not the default maps': crowded
maps, with one and two and four rects a bit of the dense list, and coordinates
far from the origin, at every lane width, against the oracle's f32 rollouts
(mantles bit for bit), which fold over every rect each time."""
import numpy as np
import pytest

from kraken_3_gpu_b200 import batch
from oracle import binding as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rects,offset", [(0, 31900.0), (0, 100000.0), (0, -650000.0), (200, 0.0), (900, 0.0),
                                          (1500, 100000.0), (3500, 0.0)])
def test_engine_equals_the_oracle(rects, offset):
    r = np.random.default_rng(rects)
    extra = np.stack([r.uniform(0, 1440, rects), r.uniform(0, 810, rects), r.uniform(3, 8, rects),
                      r.uniform(3, 8, rects)], 1)
    m = np.concatenate([ob.make_map_rects(seed=2), extra]) + np.array([offset, offset, 0, 0])
    m = m.astype(np.float32).astype(np.float64)
    n = 8
    arms, segs = np.array([6, 4, 8, 5, 1, 6, 3, 7]), np.array([7, 5, 9, 8, 1, 7, 2, 6])
    x, y = offset + r.uniform(300, 1100, n), offset + r.uniform(250, 550, n)
    angle, seed, horizon = r.uniform(0, 6, n), np.arange(n, dtype=np.uint32), np.full(n, 40)
    maps, map_id = [m], np.zeros(n, np.int32)
    _, _, ref = ob.bench_rollouts(maps, map_id, arms, segs, x, y, angle, seed, horizon, 1, metrics=True, f32=True)
    F = batch.METRIC_FIELDS
    for lanes in (32, 16, 8):
        eng = batch.BatchEngine(maps, n)
        eng.spawn(0, arms, segs, map_id, x, y, angle, horizon, seed=seed)
        eng.set_launch(4, 0, lanes_per_creature=lanes)
        eng.run(40)
        met = eng.read_metrics()
        eng.close()
        assert np.array_equal(met[:, [F.index("x"), F.index("y")]], ref[:, :2]), lanes
