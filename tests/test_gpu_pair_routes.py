"""The pair batch's routes by size: eight lanes per clone for few clones, one beyond, the same bits on both sides of the
rule; and the reductions of pairs of more than 1,024 clones (sorted to 16,384, selected beyond) against numpy's sort,
with runs of equal values and values that differ in their last bits only."""
import ctypes as C

import numpy as np
import pytest

import phygas_gb300 as pg
from tests.test_gpu_orbit32 import circular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 257])
def test_few_and_many_clones_give_the_same_bits(built, n):
    rng = np.random.default_rng(n)
    ps = np.concatenate([circular(rng, 6000), circular(rng, 400, 2.0, 0.5), circular(rng, 400, 99.0, 2.0)])
    ps[5, 0], ps[6, :3] = np.nan, [3e6, 0, 0]               # the FP64 trace among the others
    ps[7, 6:] = ps[7, :6]
    rng.shuffle(ps)
    with pg.Context(0) as ctx:
        many, clones = ctx.pair([0, len(ps)], ps.ravel(), [240], [-0.05], [900.0], [2000.0], want_clones=True)
        for a in range(0, len(ps) - n, 1 + len(ps) // 20):
            res, few = ctx.pair([0, n], ps[a:a + n].ravel(), [240], [-0.05], [900.0], [2000.0], want_clones=True)
            assert np.array_equal(few, clones[:, a:a + n], equal_nan=True), a




@pytest.mark.parametrize("m", [1025, 4096, 16383, 16384, 16385, 20000, 100003])
@pytest.mark.parametrize("kind", ["spread", "equal", "runs", "last bits", "wide"])
def test_large_reductions_are_exact(built, m, kind):
    lib = C.CDLL(pg.LIB_PATH)
    D = C.POINTER(C.c_double)
    lib.ph_pair_reduce.argtypes, lib.ph_pair_reduce.restype = [C.POINTER(pg.PhCluster), C.c_int, D, D, D,
                                                               C.POINTER(pg.PhResult)], None
    rng = np.random.default_rng(m)
    x = {"spread": lambda: rng.exponential(size=(3, m)), "equal": lambda: np.full((3, m), 0.25),
         "runs": lambda: rng.integers(0, 5, (3, m)) / 8.0,
         "last bits": lambda: 1.0 + rng.integers(0, 300, (3, m)) * 2.0 ** -52,
         "wide": lambda: 10.0 ** rng.uniform(-300, 300, (3, m))}[kind]()
    c, r = pg.PhCluster(), pg.PhResult()
    c.r50_pc, c.rtot_pc = 300.0, 1000.0
    lib.ph_pair_reduce(C.byref(c), m, *[pg._ptr(np.ascontiguousarray(v)) for v in x], C.byref(r))
    kms = 977.7922216807892
    assert r.n == m
    for name, v in zip("dtv", (x[0] * 1000.0, x[1], x[2] * kms)):
        v = np.sort(v)
        for tag, f in (("05", 0.05), ("50", 0.5), ("95", 0.95)):
            pos = f * (m - 1)
            i = int(pos)
            want = v[i] + (pos - i) * (v[i + 1] - v[i]) if i < m - 1 else v[m - 1]
            assert getattr(r, name + tag) == want, (name, tag)
    assert r.f_r50 == np.count_nonzero(x[0] * 1000.0 < 300.0) / m
    assert r.f_rtot == np.count_nonzero(x[0] * 1000.0 < 1000.0) / m
