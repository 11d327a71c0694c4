"""The clone kernel's tuner: whatever shape it keeps, small batches take eight lanes per clone with the same bits, and the
tuner compares that kernel with the shapes, on orbits of every route and pairs of every reduction."""
import numpy as np
import pytest

import phygas_gb300 as pg
from tests.test_gpu_orbit32 import circular
from tests.test_gpu_orbit32_range import clones

pytestmark = pytest.mark.gpu


def test_small_batches_after_tuning(built):
    rng = np.random.default_rng(41)
    odd = clones(rng)
    n = np.array([len(odd), 1500, 1, 33, 0, 4000])
    off = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    ps = np.concatenate([odd, circular(rng, int(off[-1]) - len(odd))])
    steps, dt = np.array([200, 100, 300, 50, 7, 120], np.int32), np.array([-0.05, -0.02, -0.1, -0.2, -0.05, -0.05])
    args = (off, ps.ravel(), steps, dt, np.full(6, 900.0), np.full(6, 2000.0))
    with pg.Context(0) as ctx:
        best, table = ctx.tune_pair(*args)
        assert 0 <= best < len(table)
        whole = ctx.pair(*args)
        for p in (0, 1, 2, 3):                       # each pair alone: a small batch
            a, b = off[p], off[p + 1]
            one = ctx.pair([0, b - a], ps[a:b].ravel(), steps[p:p + 1], dt[p:p + 1], [900.0], [2000.0])
            assert one.tobytes() == whole[p:p + 1].tobytes(), p
