"""PHYGAS_PAIR_FP64=1: a context whose clones are all traced in FP64 steps -- the same bits from few clones (four at a time by
a warp) and many (one a lane), the oracle's results to FP64's rounding, and other bits than the float pairs'."""
import numpy as np
import pytest

import phygas_gb300 as pg
from tests.test_gpu_orbit32 import circular, oracle, trace      # noqa: F401

pytestmark = pytest.mark.gpu


def test_every_clone_in_fp64(built, oracle, monkeypatch):      # noqa: F811
    rng = np.random.default_rng(51)
    ps = circular(rng, 40 * 152)
    with pg.Context(0) as ctx:
        default = trace(ctx, ps[:64], 400, -0.05)
    monkeypatch.setenv("PHYGAS_PAIR_FP64", "1")
    with pg.Context(0) as ctx:
        many = trace(ctx, ps, 400, -0.05)
        for n in (1, 4, 5, 33, 64):
            assert np.array_equal(trace(ctx, ps[:n], 400, -0.05), many[:, :n]), n
    monkeypatch.delenv("PHYGAS_PAIR_FP64")
    later = default[1] > 0                     # (half of them recede: nearest at the start, on any route)
    assert later.sum() > 8 and np.count_nonzero((many[0, :64] != default[0])[later]) > later.sum() / 2
    assert np.allclose(many[:, :64], default, rtol=1e-9, atol=1e-12)
    # distances: a difference of two positions of 8 kpc that 400 FP64 steps round by 1e-15 each
    for k in range(64):
        assert abs(many[0, k] - oracle(ps[k], 400, -0.05)[0]) <= 1e-12, k
