"""The orbit on FP32 pairs and 64-bit integers (phygas_gb300/csrc/cuda/pgx_orbit32.cuh, compiled here as host C++) is at
least as accurate as the FP64 step it stands in for: both are traced beside the same leapfrog in 113-bit arithmetic,
over 100 Myr at the default step and over the ends of the range of steps.  The fast reciprocal square root and
reciprocal are exact and at either end of the units' documented error."""
import os
import platform
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_SRC = os.path.join(REPO, "phygas_gb300", "csrc", "cuda")

HARNESS = r"""
#include <quadmath.h>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "pgx_orbit32.cuh"
using namespace pgx;
typedef __float128 Q;
constexpr double kKms = 977.7922216807892, kG = 4.30091e-6 / (kKms * kKms);
constexpr double kBulge = kG * (606.0 * 2.325e7), kB2 = 0.3873 * 0.3873, kDisk = kG * (3690.0 * 2.325e7), kA = 5.3178,
                 kD2 = 0.25 * 0.25, kHalo = kG * (4615.0 * 2.325e7), kInvA = 1.0 / 12.0, kPow = 2.02 - 1.0;
struct Model {
    static constexpr double bulge_GM = kBulge, disk_GM = kDisk, halo_GM = kHalo, halo_inv_a = kInvA;
    static constexpr double a = kPow - 1.0, s = -0.5 * a;
    static constexpr float cut2 = 1e4f, a1 = split2(s).h, a1l = split2(s).l, c2 = (float)(s * (s - 1) / 2),
                           c3 = (float)(s * (s - 1) * (s - 2) / 6), c4 = (float)(s * (s - 1) * (s - 2) * (s - 3) / 24);
    static constexpr F2 bulge_b2() { return split2(kB2); }
    static constexpr F2 disk_b2() { return split2(kD2); }
    static constexpr F2 disk_a() { return split2(kA); }
    static constexpr F3 far() { return split3(89.6846708671283); }
};
template <class T> T root(T x);
template <> double root(double x) { return sqrt(x); }
template <> Q root(Q x) { return sqrtq(x); }
template <class T> T power(T x, T y);
template <> double power(double x, double y) { return pow(x, y); }
template <> Q power(Q x, Q y) { return powq(x, y); }
template <class T> void accel(const T *p, T *a) {
    const T R2 = p[0] * p[0] + p[1] * p[1], r2 = R2 + p[2] * p[2], r = root<T>(r2), rb = r2 + (T)kB2;
    const T z = root<T>(p[2] * p[2] + (T)kD2), s = (T)kA + z, D2 = s * s + R2, x = (r < 100 ? r : (T)100) * (T)kInvA;
    const T w = power<T>(x, (T)kPow), g = -(T)kBulge / (rb * root<T>(rb)) - (T)kHalo * x * w / (1 + w) / (r2 * r);
    const T d = -(T)kDisk / (D2 * root<T>(D2));
    a[0] = (g + d) * p[0]; a[1] = (g + d) * p[1]; a[2] = p[2] * (g + d * (s / z));
}
template <class T> void step(T *p, T *v, T *a, double dt) {
    for (int c = 0; c < 3; c++) { v[c] += a[c] * (T)(0.5 * dt); p[c] += v[c] * (T)dt; }
    accel<T>(p, a);
    for (int c = 0; c < 3; c++) v[c] += a[c] * (T)(0.5 * dt);
}
int main(int, char **argv) {
    host_fast_err = (float)atof(argv[1]);
    const double dt = atof(argv[2]), size = atof(argv[4]);
    const int steps = atoi(argv[3]);
    std::vector<Halo32> halo(kHalo32N);
    for (int n = 0; n < kHalo32N; n++) halo[n] = halo32_entry(n, Model::a, kInvA);
    auto table = [&](int n) { return halo[n]; };
    std::mt19937_64 g(11);
    std::normal_distribution<double> N;
    double e64 = 0, e32 = 0;
    const int n = 60;
    for (int k = 0; k < n; k++) {
        double p[3] = {size * (-1 + 0.2 * N(g)), size * 0.3 * N(g), size * 0.05 * N(g)}, v[3], a[3];
        const double R = sqrt(p[0] * p[0] + p[1] * p[1]), sv = k % 3 == 0 ? 0.01 : (k % 3 == 1 ? 0.04 : 0.27);
        v[0] = 0.23 * p[1] / R + sv * N(g); v[1] = -0.23 * p[0] / R + sv * N(g); v[2] = 0.5 * sv * N(g);
        Q qp[3], qv[3], qa[3];
        for (int c = 0; c < 3; c++) { qp[c] = p[c]; qv[c] = v[c]; }
        accel<Q>(qp, qa);
        accel<double>(p, a);
        OrbitScale s;
        if (!orbit32_scale(4 * size + 200, dt, s)) return 2;
        const Force32 K = force32_constants<Model>(dt, s);
        Orbit32 o;
        float r2;
        orbit32_start<Model>(o, K, table, s, p, v, dt, r2);
        for (int i = 0; i < steps; i++) {
            step<Q>(qp, qv, qa, dt);
            step<double>(p, v, a, dt);
            o.x += o.wx >> 6; o.y += o.wy >> 6; o.z += o.wz >> 6;
            const Acc64i A = accel32<Model>(K, table, s.c, o.x, o.y, o.z, r2);
            o.wx += A.x; o.wy += A.y; o.wz += A.z;
        }
        const int64_t X[3] = {o.x, o.y, o.z};
        for (int c = 0; c < 3; c++) {
            const double d = (double)(p[c] - qp[c]), f = (double)((Q)X[c] * (Q)ldexp(1.0, s.e - 55) - qp[c]);
            e64 += d * d;
            e32 += f * f;
        }
    }
    printf("%.6e %.6e\n", sqrt(e64 / n), sqrt(e32 / n));
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if platform.machine() != "x86_64":
        pytest.skip("113-bit arithmetic (libquadmath) on x86 only")
    d = tmp_path_factory.mktemp("orbit32")
    src, exe = d / "h.cpp", d / "h"
    src.write_text(HARNESS)
    r = subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-I", CUDA_SRC, str(src), "-o", str(exe),
                        "-lquadmath"], stderr=subprocess.PIPE, text=True)
    if "quadmath" in r.stderr and r.returncode:
        pytest.skip("no libquadmath")
    assert r.returncode == 0, r.stderr
    return str(exe)


# orbit size (kpc): inside the bulge, the solar circle and beyond, past the halo's cut-off, in larger units.  At the
# solar circle FP64's rounding of positions near 8 kpc is the larger error by far; inside 1 kpc, where the accelerations
# are tens of times larger, the two are alike (half as much again allowed for 60 orbits' scatter).
@pytest.mark.parametrize("size,worse", [(0.5, 1.5), (3.0, 1.0), (8.0, 0.5), (30.0, 0.5), (130.0, 0.5), (400.0, 1.0)])
def test_no_larger_error_than_fp64(harness, size, worse):
    for err in ("0", "1.3e-7", "-1.3e-7"):                  # 2^-22.9: rsqrt.approx's documented error
        e64, e32 = map(float, subprocess.check_output([harness, err, "-0.05", "2000", str(size)]).split())
        assert e32 <= worse * e64, (size, err, e64, e32)


@pytest.mark.parametrize("dt,steps", [(-0.01, 1500), (-0.125, 800), (0.05, 400), (-0.05, 1)])
def test_ends_of_the_step_range(harness, dt, steps):
    e64, e32 = map(float, subprocess.check_output([harness, "0", str(dt), str(steps), "8"]).split())
    assert e32 <= e64, (dt, e64, e32)
