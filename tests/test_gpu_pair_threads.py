"""Contexts on several host threads reduce pairs whose sorts need different amounts of shared memory: no call of one may
change what a launch of the other is allowed."""
import threading

import numpy as np
import pytest

import phygas_gb300 as pg
from tests.test_gpu_orbit32 import circular

pytestmark = pytest.mark.gpu


def test_threads_with_large_pairs_of_different_sizes(built):
    sizes, rounds = (4200, 8200), 2000
    want, errors = {}, []
    for n in sizes:
        with pg.Context(0) as ctx:
            want[n] = ctx.pair([0, n], circular(np.random.default_rng(n), n).ravel(), [1], [-0.05], [10.0], [30.0])

    def work(n):
        try:
            ps = circular(np.random.default_rng(n), n).ravel()
            with pg.Context(0) as ctx:
                for _ in range(rounds):
                    if ctx.pair([0, n], ps, [1], [-0.05], [10.0], [30.0]).tobytes() != want[n].tobytes():
                        errors.append("%d clones: another result" % n)
        except Exception as e:
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(n,)) for n in 4 * sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
