"""The state-transition orbits' two kernels (four lanes per orbit for few objects, one lane beyond) give the same bits:
objects alone, ragged track lengths, and counts on both sides of the rule between them."""
import numpy as np
import pytest

import phygas_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 9, 33, 694])
def test_small_and_large_batches_give_the_same_tracks(built, golden, n):
    stars = pg.read_targets(golden["screen"])[:1100]
    ps0, sig, _ = pg.draw_targets(stars)
    ps0[5, :3] = [0.0, 0.0, 0.0]                      # the force's special case at the centre
    ps0[6, :3] = [150.0, 1.0, 2.0]                    # past the halo's cut-off
    npts = 2 + (np.arange(len(ps0)) * 7) % 40
    with pg.Context(0) as ctx:
        every = ctx.lin(ps0, sig, npts)
        few = ctx.lin(ps0[:n], sig[:n], npts[:n])
    for a, b in zip(few, every):
        assert np.array_equal(a, b[:len(a)], equal_nan=True)
