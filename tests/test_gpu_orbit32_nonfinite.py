"""Clones that are no orbit (a NaN or an infinity among their coordinates) end as the FP64 trace ends them, on both kernels,
and leave the other clones of their warps alone."""
import numpy as np
import pytest

from tests.test_gpu_orbit32 import circular, ctx, trace      # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 40 * 152], ids=["eight lanes", "one lane"])
def test_nan_and_infinite_clones(ctx, n):      # noqa: F811
    ps = circular(np.random.default_rng(6), n)
    want = trace(ctx, ps, 100, -0.05)
    bad = ps.copy()
    bad[9, 1], bad[10, 4], bad[11, 0], bad[12, 9] = np.nan, np.inf, -np.inf, np.nan
    got = trace(ctx, bad, 100, -0.05)
    keep = np.setdiff1d(np.arange(n), [9, 10, 11, 12])
    assert np.array_equal(got[:, keep], want[:, keep])
    start = np.linalg.norm(ps[:, :3] - ps[:, 6:9], axis=1)
    # a NaN position: no distance at any time, and the speed it starts with
    assert np.isnan(got[0, 9])
    assert got[1, 9] == 0.0 and abs(got[2, 9] - np.linalg.norm(ps[9, 3:6] - ps[9, 9:12])) <= 1e-15
    # an infinite speed: nothing after the start is nearer, the speed there is infinite
    assert abs(got[0, 10] - start[10]) <= 1e-15 * start[10] * 4
    assert got[1, 10] == 0.0 and np.isposinf(got[2, 10])
    # an infinite position: infinitely far at all times
    assert np.isposinf(got[0, 11])
    assert got[1, 11] == 0.0 and np.isfinite(got[2, 11])
    # a NaN speed: nothing after the start is nearer
    assert abs(got[0, 12] - start[12]) <= 1e-15 * start[12] * 4
    assert got[1, 12] == 0.0 and np.isnan(got[2, 12])
