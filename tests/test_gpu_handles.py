"""Handles over their lifetime: what closing one gives back."""
import numpy as np
import pytest

from kraken_3_gpu_b200 import batch
from oracle import binding as ob

pytestmark = pytest.mark.gpu


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
