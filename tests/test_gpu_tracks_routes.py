"""The coarse tracks' two routes: the float-pair orbit and, for orbits outside its range, the FP64 trace that overwrites what
the first one wrote -- the bits of the state-transition orbits (pgx_lin), which take the same FP64 steps.  Ordinary orbits and
such ones in the same groups of eight, tracks of one point to many."""
import numpy as np
import pytest

import phygas_gb300 as pg
from tests.test_gpu_orbit32 import circular

pytestmark = pytest.mark.gpu

# (position, velocity, points from which on the track is FP64's): at rest near the centre, far off, a NaN, one that swings
# through the centre and comes within 2^-10 kpc of it in 100 Myr, and ones inside the range at other scales
ODD = [((0.1, 0.05, 0.0), (0.0, 0.0, 0.0), 1), ((2e5, 0.0, 0.0), (0.01, 0.2, 0.0), 10000),
       ((2e6, 1.0, 0.0), (0.0, 0.0, 0.0), 1), ((1.0, 2.0, np.nan), (0.1, 0.1, 0.1), 1),
       ((0.9, 0.0, 0.0), (0.0, 0.0, 0.0), 201), ((150.0, 3.0, 2.0), (0.0, 0.1, 0.0), 10000),
       ((900.0, 3.0, 2.0), (0.0, 0.1, 0.0), 10000), ((3.0, 0.1, 0.0), (0.0, 0.02, 0.01), 10000)]


@pytest.fixture(scope="module")
def ctx(built):
    with pg.Context(0) as c:
        yield c


@pytest.mark.parametrize("n", [1, 7, 8, 9, 21])
@pytest.mark.parametrize("first", [0, 3, 5])
def test_tracks_of_both_routes(ctx, n, first):
    rng = np.random.default_rng(31)
    ps = circular(rng, n)[:, :6]
    npts = np.array([(1, 30, 2, 201, 57)[k % 5] for k in range(n)], np.int32)
    if n == 1:
        npts[0] = 201
    fp64 = np.zeros(n, bool)
    for k in range(0, n, 2):                         # every other object an odd one
        p, v, points = ODD[(first + k // 2) % len(ODD)]
        ps[k], fp64[k] = p + v, npts[k] >= points
    got = ctx.tracks(ps, npts)
    want = ctx.lin(ps, np.zeros((n, 6, 6)), npts)[0]
    off = np.concatenate([[0], np.cumsum(npts)])
    for k in range(n):
        a, b = got[off[k]:off[k + 1]], want[off[k]:off[k + 1]]
        if fp64[k]:
            assert np.array_equal(a, b, equal_nan=True), k
        else:
            assert np.array_equal(a[0], ps[k, :3]) and np.abs(a - b).max() < 1e-9, (k, np.abs(a - b).max())


def test_an_orbit_that_leaves_the_range_late(ctx):
    ps = circular(np.random.default_rng(32), 9)[:, :6]
    ps[4] = [15.0, 1.0, 1.0, 0.39, 0.39, 0.39]       # unbound: past 256 kpc after some 500 Myr
    npts = np.full(9, 21, np.int32)
    npts[4] = 1601
    off = np.concatenate([[0], np.cumsum(npts)])
    got = ctx.tracks(ps, npts)
    want = ctx.lin(ps, np.zeros((9, 6, 6)), npts)[0]
    assert np.linalg.norm(want[off[5] - 1]) > 260.0
    assert np.array_equal(got[off[4]:off[5]], want[off[4]:off[5]])
    assert np.abs(got - want).max() < 1e-9
