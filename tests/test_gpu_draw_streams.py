"""The device's clone draws where tries fail: a parallax or a distance drawn again moves every later clone of the pair
along the random stream, and a clone whose tries all fail is dropped.  Against the host's draws (the reference's): the
same clones succeed and the same streams are taken, values within the device math functions' last bits."""
import numpy as np
import pytest

import phygas_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_clones", [0, 1, 31, 32, 33, 257])
def test_failing_tries_match_the_host(built, golden, n_clones):
    clusters = pg.read_clusters(golden["clusters"])
    stars, pulsars = pg.read_targets(golden["screen"]), pg.read_targets(golden["pulsar"])
    nt = 8
    t = (pg.PhTarget * nt)(*([stars[k] for k in range(nt - 1)] + [pulsars[0]]))
    c = (pg.PhCluster * nt)(*[clusters[k] for k in range(nt)])
    t[0].e_plx = 0.5 * t[0].plx                # one try in 44 fails
    t[1].e_plx = 30.0 * t[1].plx               # about half
    t[2].e_plx = -0.4 * t[2].plx
    t[3].e_plx = 0.0
    t[4].plx, t[4].e_plx = 1e-6, 1e6
    t[5].plx, t[5].dist_pc, t[5].e_lndist = -1.0, 800.0, 0.25
    t[6].plx, t[6].dist_pc = 0.0, -5.0         # every try fails: no clone
    c[1].e_dist_pc = 0.7 * c[1].dist_pc
    c[2].dist_pc, c[2].e_dist_pc = -1.0, 0.5   # one try in 44 succeeds: some clones fail all fifty
    c[3].e_dist_pc = 0.0
    ti, ci = [a.ravel().astype(np.int32) for a in np.meshgrid(np.arange(nt), np.arange(nt), indexing="ij")]
    n = np.full(len(ti), n_clones, np.int32)
    n[::7] = n_clones // 2
    want = pg.draw_pair_batch(t, ti, c, ci, n)
    with pg.Context(0) as ctx:
        got = ctx.draw_pair_batch(t, ti, c, ci, n)
    assert np.array_equal(got[0], want[0])
    if n_clones >= 257:
        assert np.diff(want[0])[ti == 6].max() == 0 and 0 < np.diff(want[0])[(ti == 0) & (ci == 2)][0] < 257
    a, b = got[1].reshape(-1, 12), want[1].reshape(-1, 12)
    for o in (0, 3, 6, 9):                     # positions and speeds: a vector's components share its rounding
        size = np.linalg.norm(b[:, o:o + 3], axis=1, keepdims=True) + 10.0
        assert np.all(np.abs(a[:, o:o + 3] - b[:, o:o + 3]) <= 1e-13 * size)
    for x, y in zip(got[2:], want[2:]):
        assert np.array_equal(x, y)
