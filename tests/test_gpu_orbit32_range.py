"""The float-pair orbit's ranges on the GPU: orbits whose steps near the centre take the bulge in FP64, orbits that start there
or so near the centre that they are FP64 throughout, the units (small, large and fast orbits, short steps) and the reach's end, against
the oracle's ph_pair_clone and with the same bits from one lane and eight lanes per clone."""
import numpy as np
import pytest

import phygas_gb300 as pg
from tests import oracle_tools as ot
from tests.test_gpu_orbit32 import circular, ctx, oracle, trace      # noqa: F401

pytestmark = pytest.mark.gpu


def clones(rng):
    """Circular and plunging orbits, fast and distant ones, and starts on both sides of the near field's radius."""
    out = [circular(rng, 8), circular(rng, 6, 1.2, 0.3), circular(rng, 6, 2.5, 0.3), circular(rng, 6, 0.4, 0.2),
           circular(rng, 4, 0.16, 0.02), circular(rng, 4, 300.0, 1.0), circular(rng, 4, 1500.0, 1.0),
           circular(rng, 4, 2e5, 1.0), circular(rng, 2, 7e5, 1.0)]
    plunge = circular(rng, 10, 3.0, 0.5)
    plunge[:, 3:6] *= 0.05
    plunge[::2, 9:12] *= 0.02
    rest = circular(rng, 6, 1.5, 0.2)
    rest[:, 3:6] = rest[:, 9:12] = 0.0
    fast = circular(rng, 6)
    fast[:, 3:6] *= np.array([2.0, 8.0, 12.0, 20.0, 40.0, 100.0])[:, None]
    return np.concatenate(out + [plunge, rest, fast])


@pytest.mark.parametrize("steps,dt", [(400, -0.05), (300, -0.01), (300, -0.0156), (300, -0.02), (300, 0.0625), (300, -0.1),
                                      (300, -0.125)])
def test_clones_match_the_oracle(ctx, oracle, steps, dt):      # noqa: F811
    ps = clones(np.random.default_rng(11))
    got = trace(ctx, ps, steps, dt)
    for k in range(len(ps)):
        o = oracle(ps[k], steps, dt)
        size = 1.0 + np.abs(ps[k]).max()
        for a, b in zip(got[:, k], o):
            assert abs(a - b) <= ot.REL_TOL * abs(b) + 1e-11 * size, (k, got[:, k], o)


@pytest.mark.parametrize("dt", [-0.05, -0.01, -0.02, -0.1])
def test_one_and_eight_lanes_give_the_same_bits(ctx, dt):      # noqa: F811
    rng = np.random.default_rng(12)
    ps = clones(rng)
    many = np.concatenate([ps, circular(rng, 40 * 152 - len(ps))])
    want = trace(ctx, many, 250, dt)[:, :len(ps)]
    assert np.array_equal(trace(ctx, ps, 250, dt), want)
    for n in (1, 3, 5):
        for a in range(0, len(ps) - n, 7):
            assert np.array_equal(trace(ctx, ps[a:a + n], 250, dt), want[:, a:a + n]), (n, a)
