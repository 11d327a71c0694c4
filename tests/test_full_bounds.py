"""The mixed filter's full bounds (point_bound32 in phygas_gb300/csrc/cuda/pgx_bounds32.cuh) on the CPU, the header compiled
as host C++ with the fast reciprocal and square root at either end of their documented error band and exact: the chi2 of a
point, evaluated as the FP64 path does (adjugate, the segment's start and its nearest point), lies within [lb, ub], and above
the cut where the trace bound rejects the point.  The points of the point test's own check, with steps that vanish and
separations and matrices scaled over twelve decades added."""
import os
import subprocess
import tempfile

import numpy as np
import pytest

from tests import test_point_bound as pb

F = np.float32

HARNESS = pb.HARNESS[:pb.HARNESS.index("        putchar(")] + r"""
        pgx::Bound b = {0.f, 0.f};
        const bool kept = pgx::point_bound32(St, Sc, p[12], p[13], m0, m1, true, p[20], b);
        const float o[3] = {kept ? 1.f : 0.f, b.lb, b.ub};
        fwrite(o, 4, 3, stdout);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness():
    d = tempfile.mkdtemp(prefix="phygas_fb_")
    src, exe = os.path.join(d, "h.cpp"), os.path.join(d, "h")
    with open(src, "w") as f:
        f.write(pb.PRELUDE + HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", pb.CUDA_SRC, src, "-o", exe], check=True)
    return exe, d


def _chi2(M, m0, m1):
    a00, a01, a02 = M[:, 1, 1] * M[:, 2, 2] - M[:, 1, 2] ** 2, M[:, 0, 2] * M[:, 1, 2] - M[:, 0, 1] * M[:, 2, 2], \
        M[:, 0, 1] * M[:, 1, 2] - M[:, 0, 2] * M[:, 1, 1]
    a11, a12, a22 = M[:, 0, 0] * M[:, 2, 2] - M[:, 0, 2] ** 2, M[:, 0, 1] * M[:, 0, 2] - M[:, 0, 0] * M[:, 1, 2], \
        M[:, 0, 0] * M[:, 1, 1] - M[:, 0, 1] ** 2
    det = M[:, 0, 0] * a00 + M[:, 0, 1] * a01 + M[:, 0, 2] * a02

    def form(x):
        return (x[:, 0] * (a00 * x[:, 0] + a01 * x[:, 1] + a02 * x[:, 2])
                + x[:, 1] * (a01 * x[:, 0] + a11 * x[:, 1] + a12 * x[:, 2])
                + x[:, 2] * (a02 * x[:, 0] + a12 * x[:, 1] + a22 * x[:, 2])) / det
    dr = m1 - m0
    dd = (dr * dr).sum(1)
    s = np.clip(-(m0 * dr).sum(1) / np.where(dd > 0, dd, 1.0), 0.0, 1.0) * (dd > 0)
    q, qs = form(m0), form(m0 + dr * s[:, None])
    return np.where((qs >= 0) & (qs < q), qs, q), det


@pytest.mark.parametrize("err", [0.0, 4 * 5.96e-8, -4 * 5.96e-8])
def test_the_chi2_lies_within_the_bounds(harness, err):
    rec, _ = pb._points(200_000, 47)
    rng = np.random.default_rng(48)
    still = rng.uniform(size=len(rec)) < 0.05
    rec[still, 17:20] = rec[still, 14:17]
    scale = np.where(rng.uniform(size=len(rec)) < 0.5, 1.0, 4.0 ** rng.integers(-10, 10, len(rec))).astype(F)
    rec[:, :14] *= (scale * scale)[:, None]                # powers of two: the same points in other units
    rec[:, 14:20] *= scale[:, None]
    exe, d = harness
    path = os.path.join(d, "in.bin")
    rec.tofile(path)
    out = np.frombuffer(subprocess.run([exe, repr(err), path], stdout=subprocess.PIPE, check=True).stdout, F)
    kept, lb, ub = out.reshape(-1, 3).T.astype(np.float64)
    r = rec.astype(np.float64)
    v, det = _chi2(pb._unpack6(r[:, 0:6] + r[:, 6:12]), r[:, 14:17], r[:, 17:20])
    ok = (det > 0) & (v >= 0)
    assert ok.mean() > 0.99
    assert np.all(v[ok & (kept == 0)] > r[ok & (kept == 0), 20])
    k = ok & (kept == 1)
    assert np.all(lb[k] <= v[k]) and np.all(v[k] <= ub[k]), (np.max(lb[k] / v[k]), np.min(ub[k] / v[k]))
    assert np.isfinite(ub[k]).mean() > 0.5
