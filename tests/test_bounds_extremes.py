"""The FP32 tests of the mixed screen (phygas_gb300/csrc/cuda/pgx_bounds32.cuh, compiled here as host C++ with the fast
units' flushing) where their reciprocals leave the normal range: separations and covariances far beyond any orbit's must
leave a point undecided, not settle it wrongly."""
import os
import subprocess

import pytest

CUDA_SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phygas_gb300", "csrc", "cuda")

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
struct float4 { float x, y, z, w; };
#include "pgx_bounds32.cuh"
using namespace pgx;
int main(int, char **argv) {
    const float len = (float)atof(argv[1]), lam = (float)atof(argv[2]), tr = (float)atof(argv[3]), off = (float)atof(argv[4]);
    // a step of length len through the origin, and the covariance diag(lam, lam, tr - 2 lam) turned into its direction
    const float m0[3] = {-0.5f * len, 0.f, off}, m1[3] = {0.5f * len, 0.f, off}, S[6] = {0.5f * lam, 0, 0, 0.5f * lam, 0, 0.5f * (tr - 2 * lam)};
    Bound b{-1.f, -1.f};
    const bool skip = point_skip32(S, S, 0.5f * lam, 0.5f * lam, m0, m1, 25.f);
    const bool keep = point_bound32(S, S, 0.5f * lam, 0.5f * lam, m0, m1, true, 25.f, b);
    const float4 t[4] = {{len / 2, 0, 0, 0}, {0, 0, 0, 0.5f * lam}, {S[0], S[1], S[2], S[3]}, {S[4], S[5], 0.5f * lam, 0}};
    const float4 c[4] = {{-len / 2, 0, 0, 0}, {0, 0, 0, 0.5f * lam}, {S[0], S[1], S[2], S[3]}, {S[4], S[5], 0.5f * lam, 0}};
    const float mid[3] = {0.3f * len, 0.f, off};
    printf("%d %d %g %g %d\n", skip, keep, b.lb, b.ub, block_skip32(t, c, mid, 25.f));
    return 0;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("extremes")
    src, exe = d / "e.cpp", d / "e"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-I", CUDA_SRC, str(src), "-o", str(exe)], check=True)

    def go(*args):
        skip, keep, lb, ub, block = subprocess.check_output([str(exe)] + [repr(float(a)) for a in args]).split()
        return int(skip), int(keep), float(lb), float(ub), int(block)
    return go


# the step passes the origin: its smallest form is 0 (or off^2 / (tr - 2 lam), under the cut), so nothing may be settled;
# the lengths take |d|^2 / lam through 2^126 to infinity
@pytest.mark.parametrize("lam", [1e-6, 1.0, 1e4])
@pytest.mark.parametrize("q", [1e30, 8e37, 8.6e37, 1.2e38, 2e38, 3.3e38, 1e39, 1e41])
def test_a_step_through_the_origin_is_never_settled(run, lam, q):
    skip, keep, lb, ub, block = run((q * lam) ** 0.5, lam, 3 * lam, 0.0)
    assert not skip and not block
    assert keep and lb <= 25.0 and ub >= 0.0, (lb, ub)


# covariances whose determinant or smallest eigenvalue leaves the range: the FP64 path's own rounding, 2.85e-14 tr^3 / det of
# its value, is then beyond any bound (det = lam^2 (tr - 2 lam)) or is not known to FP32
@pytest.mark.parametrize("lam,tr", [(1e10, 1e19), (1e12, 1e21), (1e13, 1e20), (1e18, 1e25), (1e3, 1e33)])
def test_covariances_beyond_the_range_are_left_open(run, lam, tr):
    skip, keep, lb, ub, block = run(1e3, lam, tr, 1e6)
    assert not skip and not block
    assert keep and lb == 0.0 and ub == float("inf"), (lb, ub)
