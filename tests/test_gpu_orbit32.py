"""The clone Monte Carlo's two routes: the FP32 orbit (pgx_orbit32.cuh) and the FP64 trace for what it does not cover,
lane by lane or by a whole warp.  Clones at the edges of the routes against the oracle's ph_pair_clone, and the two
forms of the FP64 trace against each other bit for bit."""
import ctypes as C

import numpy as np
import pytest

import phygas_gb300 as pg
from tests import oracle_tools as ot

pytestmark = pytest.mark.gpu
D = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def ctx(built):
    c = pg.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def oracle(built):
    L = C.CDLL(ot.ORACLE_LIB)
    L.ph_pair_clone.argtypes, L.ph_pair_clone.restype = [D, C.c_int, C.c_double, D, D, D], None
    L.ph_init()

    def clone(ps, steps, dt):
        out = [C.c_double() for _ in range(3)]
        L.ph_pair_clone(pg._ptr(np.ascontiguousarray(ps)), steps, dt, *[C.byref(x) for x in out])
        return [x.value for x in out]
    return clone


def circular(rng, n, size=8.1, spread=0.05):
    """n clones: a target and a cluster near each other on disk orbits of about `size` kpc."""
    ps = np.zeros((n, 12))
    for o in (0, 6):
        p = np.array([-size, 0.1, 0.02]) + spread * rng.normal(size=(n, 3))
        R = np.hypot(p[:, 0], p[:, 1])
        ps[:, o:o + 3] = p
        ps[:, o + 3:o + 6] = np.stack([0.23 * p[:, 1] / R, -0.23 * p[:, 0] / R, 0 * R], 1) + 0.03 * rng.normal(size=(n, 3))
    return ps


def trace(ctx, ps, steps, dt):
    n = len(ps)
    res, clones = ctx.pair([0, n], ps.ravel(), [steps], [dt], [10.0], [30.0], want_clones=True)
    assert res["n"][0] == n
    return clones


# inside and outside the FP32 orbit's step lengths and reach (units of 1, 2, 4, ... 2^11 times 2^-55 kpc, then FP64),
# through the Galactic centre (inside 2^-10 kpc: FP64) and past the halo's cut-off at 100 kpc
@pytest.mark.parametrize("name,size,steps,dt", [
    ("default", 8.1, 400, -0.05), ("shortest", 8.1, 300, -0.01), ("below", 8.1, 300, -0.0099), ("longest", 8.1, 300, -0.125),
    ("above", 8.1, 300, -0.1251), ("forward", 8.1, 300, 0.05), ("one step", 8.1, 1, -0.05), ("cut-off", 100.0, 300, -0.05),
    ("unit 2", 150.0, 300, -0.05), ("unit 2^11", 2e5, 300, -0.05), ("far", 2e6, 300, -0.05), ("inner", 0.3, 400, -0.05),
    ("centre", 0.001, 40, -0.05)])
def test_clones_at_the_edges_match_the_oracle(ctx, oracle, name, size, steps, dt):
    ps = circular(np.random.default_rng(3), 37, size, 0.05 * min(size, 1.0))
    if name == "centre":
        ps[:, 3:6] = ps[:, 9:12] = 0.0
        ps[:, 0:3] *= 0.5                      # falls through within 2^-10 kpc
    got = trace(ctx, ps, steps, dt)
    for k in range(len(ps)):
        o = oracle(ps[k], steps, dt)
        for a, b in zip(got[:, k], o):
            assert abs(a - b) <= ot.REL_TOL * abs(b) + 1e-12 * size, (name, k, got[:, k], o)


def test_odd_clones_match_the_oracle(ctx, oracle):
    """Co-moving, coincident and receding pairs, a pair at rest, and one clone beyond the reach in a warp of others."""
    ps = circular(np.random.default_rng(5), 40)
    ps[3, 6:] = ps[3, :6]                      # the same orbit: separation 0
    ps[4, 6:] = ps[4, :6] + np.array([1e-3, 0, 0, 0, 0, 0])
    ps[5, 9:] = ps[5, 3:6]
    ps[6, 3:6] = ps[6, 9:12] = 0.0
    ps[7, :3] = [3e6, 0.0, 0.0]
    ps[8, 3:6] = [40.0, 0.0, 0.0]
    got = trace(ctx, ps, 500, -0.05)
    for k in range(len(ps)):
        o = oracle(ps[k], 500, -0.05)
        for a, b in zip(got[:, k], o):
            assert abs(a - b) <= ot.REL_TOL * abs(b) + 1e-11, (k, got[:, k], o)


def test_nan_and_infinite_clones_trace_as_fp64(ctx):
    """Clones that are no orbit leave the others alone, and end as the FP64 trace ends: the separation they start at."""
    ps = circular(np.random.default_rng(6), 33)
    want = trace(ctx, ps, 100, -0.05)
    bad = ps.copy()
    bad[9, 1], bad[10, 4], bad[11, 0] = np.nan, np.inf, -np.inf
    got = trace(ctx, bad, 100, -0.05)
    keep = [k for k in range(33) if k not in (9, 10, 11)]
    assert np.array_equal(got[:, keep], want[:, keep])
    assert np.isnan(got[0, 9]) and np.isinf(got[0, 11]) and got[0, 10] == want[0, 10] or not np.isfinite(got[2, 10])


@pytest.mark.parametrize("n", [1, 4])
def test_warp_and_lane_fp64_traces_give_the_same_bits(ctx, n):
    """A step length outside the FP32 orbit's: up to four clones of a warp are traced by the whole warp (four lanes an
    orbit), more lane by lane -- the same operations, the same bits.  Orbits through the centre and past the cut-off
    take the force's special cases."""
    rng = np.random.default_rng(8)
    ps = np.concatenate([circular(rng, 12), circular(rng, 12, 0.4), circular(rng, 12, 99.0),
                         circular(rng, 12, 1e3, 1e-3)])
    ps[3, :6] = [0.3, 0.0, 0.0, 0.0, 0.0, 0.0]           # straight through the centre
    ps[4, :6] = [1e-13, 0.0, 0.0, 0.0, 0.0, 0.0]
    every = trace(ctx, ps, 300, -0.2)
    for k in range(0, len(ps), n):
        assert np.array_equal(trace(ctx, ps[k:k + n], 300, -0.2), every[:, k:k + n]), k
