"""The clone's FP64 trace: up to twelve clones of a warp are traced four at a time, eight lanes each, more lane by lane --
the same bits, whatever the number of them in a warp, beside clones of the float-pair orbit, and on both kernels (few
clones: eight lanes each; many: one)."""
import numpy as np
import pytest

from tests.test_gpu_orbit32 import circular, ctx, trace      # noqa: F401

pytestmark = pytest.mark.gpu
MANY = 40 * 152                                  # above the number that takes eight lanes per clone


@pytest.mark.parametrize("dt", [-0.05, -0.2])
def test_any_number_of_them_in_a_warp(ctx, dt):      # noqa: F811
    rng = np.random.default_rng(21)
    inner = circular(rng, 64, 0.08, 0.01)        # FP64 at any step
    inner[3, :6] = [0.12, 0.0, 0.0, 0.0, 0.0, 0.0]
    inner[4, :6] = [1e-13, 0.0, 0.0, 0.0, 0.0, 0.0]
    inner[5, :3], inner[6, :3] = [150.0, 1.0, 2.0], [3e6, 0.0, 0.0]
    alone = np.concatenate([trace(ctx, inner[k:k + 1], 200, dt) for k in range(64)], axis=1)
    for n in (2, 3, 4, 5, 32, 64):               # the kernel of few clones
        assert np.array_equal(trace(ctx, inner[:n], 200, dt), alone[:, :n]), n
    ps = circular(rng, MANY)
    for w, n in enumerate((1, 3, 4, 5, 8, 9, 12, 13, 31, 32)):      # warp w: n of them, spread over its lanes
        ps[32 * w + np.sort(rng.permutation(32)[:n])] = inner[:n]
    got = trace(ctx, ps, 200, dt)
    for w, n in enumerate((1, 3, 4, 5, 8, 9, 12, 13, 31, 32)):
        mine = [k for k in range(32 * w, 32 * w + 32) if np.abs(ps[k, 6:9]).max() < 1.0]
        assert len(mine) == n and np.array_equal(got[:, mine], alone[:, :n]), (w, n)
