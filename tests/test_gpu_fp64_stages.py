"""The FP64 screen's stages at their edges: the scan's queue and its FP32 trace test (star counts around the warp and
block, cuts with and without the test), and the draws' three stages for pairs of every kind against the oracle."""
import ctypes as C

import numpy as np
import pytest

import phygas_gb300 as pg
from tests import oracle_tools as ot
from tests import test_gpu_dropin as dropin

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def data(golden):
    return pg.read_clusters(golden["clusters"])[:257], pg.read_targets(golden["screen"])[:200]


def test_star_counts_and_cuts(built, data):
    clusters, stars = data
    tmax = max(c.tmax_myr for c in clusters)
    with pg.Context(0) as ctx:
        ctx.set_clusters(clusters)
        draws = pg.draw_targets(stars)
        for cut in (1e-3, 25.0, 1e4):
            every = ctx.screen(*draws, tmax, cut, pg.PGX_FP64)
            for n in (1, 31, 32, 33, 128, 129):
                rows = ctx.screen(*[a[:n] for a in draws], tmax, cut, pg.PGX_FP64)
                assert np.array_equal(rows, every[every["star"] < n]), (cut, n)
        # beyond 1e30 the trace test runs in FP64, an infinite cut has none: every pair's minimum is the same
        few = [a[:40] for a in draws]
        a, b, c = [ctx.screen(*few, tmax, cut, pg.PGX_FP64) for cut in (9e29, 2e30, np.inf)]
        assert np.array_equal(a, b) and np.array_equal(a, c) and len(a) == 40 * len(clusters)


def test_draw_stages_match_the_oracle(built, data):
    """ph_screen_finish on made-up tracks: separations from inside both radii to far outside, along every axis; radii
    zero, equal and wide; covariances isotropic, needles along x and across it, singular and zero."""
    gpu, ora = dropin._bind(pg.LIB_PATH), dropin._bind(ot.ORACLE_LIB)
    rng = np.random.default_rng(4)
    base = data[0][3]
    checked = inside = 0
    for case in range(400):
        sig = 10.0 ** rng.uniform(-3, 0)
        L = np.tril(rng.normal(size=(3, 3))) * sig
        if case % 5 == 1:
            L[:, 0] *= 30.0
        if case % 5 == 2:
            L[:, 0] *= 1e-4
        if case % 5 == 3:
            L[2] = L[1]
        if case % 25 == 4:
            L[:] = 0.0
        S = L @ L.T
        S6 = np.array([[S[0, 0], S[0, 1], S[0, 2], S[1, 1], S[1, 2], S[2, 2]]])
        sep = rng.normal(size=3) * sig * rng.choice([0.0, 0.3, 1.0, 3.0])
        if case % 7 == 0:
            sep[1:] = 0.0
        pos_c = np.array([[-8.0, 0.3, 0.05]])
        lins = []
        for p, s in ((pos_c + sep, S6), (pos_c, 0 * S6)):
            l = dropin.PhLin()
            l.n = 1
            keep = [np.ascontiguousarray(p), np.zeros((1, 3)), np.ascontiguousarray(s)]
            for name, a in zip(("pos", "vel", "S"), keep):
                kind = dict(dropin.PhLin._fields_)[name]
                setattr(l, name, C.cast(a.ctypes.data, kind))
            lins.append((l, keep))
        c = pg.PhCluster()
        C.memmove(C.byref(c), C.byref(base), C.sizeof(c))
        c.r50_pc = 1000.0 * sig * rng.choice([0.0, 0.05, 0.5, 3.0, 30.0])
        c.rtot_pc = c.r50_pc * rng.choice([0.5, 1.0, 3.0])
        got = []
        for lib in (gpu, ora):
            r = dropin.PhScreen()
            lib.ph_screen_finish(C.byref(lins[0][0]), C.byref(lins[1][0]), C.byref(c), 1234567 + case, 1.0, 0, 0.0,
                                 C.byref(r))
            got.append((r.p_r50, r.p_rtot))
        # a draw within rounding of a radius may fall either way; one with no spread lies at the separation itself
        assert np.allclose(got[0], got[1], atol=1.5 / 512 if case % 25 == 4 else 0.0, rtol=0.0), (case, got)
        checked += 1
        inside += 0 < got[0][0] < 1
    assert checked == 400 and inside > 40, inside


@pytest.mark.parametrize("precision", [pg.PGX_FP64, pg.PGX_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("cut,r_kernel", [(25.0, 2.0), (4.0, 0.0), (400.0, 8.0)])
def test_classified_points_give_the_general_paths_bits(built, data, precision, cut, r_kernel):
    """The points that the FP32 classification rejects or shortens: the batched screens' chi2, argmin and segment fraction
    against one pair at a time, whose points all take the whole FP64 evaluation, on the same tracks bit for bit."""
    clusters, stars = data[0][:64], data[1][:20]
    gpu = dropin._bind(pg.LIB_PATH)
    C.c_double.in_dll(gpu, "ph_screen_r").value = r_kernel
    tmax = max(c.tmax_myr for c in clusters)
    t0, c0 = pg.draw_targets(stars), pg.draw_clusters(clusters)
    nt = int(np.ceil(tmax / 0.5)) + 1
    cn = [int(np.ceil(c.tmax_myr / 0.5)) + 1 for c in clusters]
    with pg.Context(0) as ctx:
        ctx.set_clusters(clusters, r_kernel=r_kernel, draws=c0)
        rows = {(int(r["star"]), int(r["cluster"])): r for r in ctx.screen(*t0, tmax, cut, precision)}
        lins = []
        for n, ps0, sig in (([nt] * len(t0[0]), t0[0], t0[1]), (cn, c0[0], c0[1])):
            pos, vel, S = ctx.lin(ps0, sig, n)
            off = np.concatenate([[0], np.cumsum(n)])
            out = []
            for i in range(len(n)):
                l = dropin.PhLin()
                l.n = n[i]
                keep = [np.ascontiguousarray(a[off[i]:off[i + 1]]) for a in (pos, vel, S)]
                for name, a in zip(("pos", "vel", "S"), keep):
                    setattr(l, name, C.cast(a.ctypes.data, dict(dropin.PhLin._fields_)[name]))
                out.append((l, keep))
            lins.append(out)
    kept = 0
    for j in range(len(stars)):
        for i in range(len(clusters)):
            kb, sb = C.c_int(), C.c_double()
            q = gpu.ph_screen_chi2_cut(C.byref(lins[0][j][0]), C.byref(lins[1][i][0]), C.byref(clusters[i]), cut,
                                       C.byref(kb), C.byref(sb))
            assert (q < cut) == ((j, i) in rows), (j, i, q)
            if q < cut:
                r = rows[(j, i)]
                assert (r["chi2"], r["kb"], r["sb"]) == (q, kb.value, sb.value), (j, i)
                kept += 1
    assert kept > 0
