"""What the float-pair orbit (phygas_gb300/csrc/cuda/pgx_orbit32.cuh) accepts comes out no further from exact arithmetic than
FP64 steps: traced beside the same leapfrog in 113-bit arithmetic over 2,000 steps, at the ends of the ranges of step, size
and reach, on ordinary orbits, circular ones, ones that plunge through the centre (whose steps near it take the bulge's
force in FP64) and ones that start at rest; and what it does not accept is refused."""
import subprocess

import pytest

from tests.test_orbit32 import CUDA_SRC, HARNESS, harness      # noqa: F401  (harness: skips where 113 bits are missing)

MAIN = r"""
// the FP64 step with its products and sums fused, as the device code has them
void step64(double *p, double *v, double *a, double dt) {
    for (int c = 0; c < 3; c++) { v[c] = fma(a[c], 0.5 * dt, v[c]); p[c] = fma(v[c], dt, p[c]); }
    accel<double>(p, a);
    for (int c = 0; c < 3; c++) v[c] = fma(a[c], 0.5 * dt, v[c]);
}
int main(int, char **argv) {
    host_fast_err = (float)atof(argv[1]);
    const double dt = atof(argv[2]), size = atof(argv[3]);
    const int kind = atoi(argv[4]), steps = 2000, n = 40;
    std::vector<Halo32> halo(kHalo32N);
    for (int k = 0; k < kHalo32N; k++) halo[k] = halo32_entry(k, Model::a, kInvA);
    auto table = [&](int k) { return halo[k]; };
    auto bulge = [](double r2) { const double i = 1.0 / sqrt(r2 + kB2); return (i * i) * (i * -kBulge); };
    auto near = [&](const Force32 &K, const OrbitScale &s, double h, int64_t x, int64_t y, int64_t z) {
        return accel_near<Model>(K, table, bulge, s, h, x, y, z);
    };
    const float near2 = orbit32_near2(dt);
    std::mt19937_64 g(3);
    std::normal_distribution<double> N;
    double e64 = 0, e32 = 0;
    std::vector<double> ratio;
    int refused = 0;
    for (int k = 0; k < n; k++) {
        double p[3] = {-size * (1 + 0.2 * fabs(N(g))), size * 0.3 * N(g), size * 0.05 * N(g)}, v[3], a[3];
        const double R = sqrt(p[0] * p[0] + p[1] * p[1]);
        const double f = kind == 1 ? 0.03 * N(g) : (kind == 3 ? 0.0 : 0.23);
        const double sv = kind == 0 ? (k % 3 == 0 ? 0.01 : (k % 3 == 1 ? 0.04 : 0.27)) : (kind == 1 ? 0.02 : (kind == 2 ? 0.01 : 0.001));
        v[0] = f * p[1] / R + sv * N(g); v[1] = -f * p[0] / R + sv * N(g); v[2] = 0.5 * sv * N(g);
        OrbitScale s;
        double vdt;
        const double reach = orbit32_reach(p, v, steps, dt, vdt);
        if (!orbit32_start_ok(p) || !orbit32_units(reach, vdt, dt, s)) { refused++; continue; }
        Q qp[3], qv[3], qa[3];
        for (int c = 0; c < 3; c++) { qp[c] = p[c]; qv[c] = v[c]; }
        accel<Q>(qp, qa);
        accel<double>(p, a);
        const Force32 K = force32_constants<Model>(dt, s);
        Orbit32 o;
        float r2;
        auto at = [&](int64_t x, int64_t y, int64_t z, float &r) {
            return orbit32_accel<Model>(K, table, near, s, dt, near2, x, y, z, r);
        };
        orbit32_start(o, at, s, p, v, dt, r2);
        const int sh = 6 + s.k;
        bool out = false;
        for (int i = 0; i < steps; i++) {
            step<Q>(qp, qv, qa, dt);
            step64(p, v, a, dt);
            o.x += o.wx >> sh; o.y += o.wy >> sh; o.z += o.wz >> sh;
            const Acc64i A = at(o.x, o.y, o.z, r2);
            o.wx += A.x; o.wy += A.y; o.wz += A.z;
            if (!(r2 < orbit32_max_r2(s))) return 3;
            out = out || !(r2 > kOrbit32MinR2);
        }
        if (out) continue;                                    // (within 2^-10 kpc of the centre: traced in FP64)
        const int64_t X[3] = {o.x, o.y, o.z};
        double d2 = 0, f2 = 0;
        for (int c = 0; c < 3; c++) {
            const double d = (double)(p[c] - qp[c]), e = (double)((Q)X[c] * (Q)ldexp(1.0, s.e - 55) - qp[c]);
            d2 += d * d;
            f2 += e * e;
        }
        e64 += d2;
        e32 += f2;
        ratio.push_back(sqrt(f2 / d2));
    }
    std::sort(ratio.begin(), ratio.end());
    printf("%d %.6e %.6e %.6e\n", refused, sqrt(e64 / n), sqrt(e32 / n), ratio.empty() ? 0.0 : ratio[ratio.size() / 2]);
    return 0;
}
"""


@pytest.fixture(scope="module")
def run(harness, tmp_path_factory):      # noqa: F811
    d = tmp_path_factory.mktemp("orbit32_range")
    src, exe = d / "r.cpp", d / "r"
    src.write_text("#include <algorithm>\n" + HARNESS[:HARNESS.index("int main(")] + MAIN)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-mfma", "-I", CUDA_SRC, str(src), "-o", str(exe),
                    "-lquadmath"], check=True)

    def go(dt, size, kind, err=0.0):
        refused, *e = subprocess.check_output([str(exe), repr(err), repr(dt), repr(size), str(kind)]).split()
        return int(refused), *map(float, e)
    return go


# (step, size): the nearest accepted start, both sides of the near field, the solar circle, the halo's cut-off, and up to the
# largest accepted reach; at the default step, the ends of the range and the steps between which the displacements' unit
# changes
@pytest.mark.parametrize("kind", [0, 2], ids=["ordinary", "circular"])
@pytest.mark.parametrize("dt,size", [(-0.01, 0.16), (-0.01, 0.42), (-0.011, 8.0), (-0.0111, 0.42), (0.03, 8.0), (-0.05, 0.16),
                                     (-0.05, 0.65), (-0.05, 8.0), (-0.05, 100.0), (-0.05, 1500.0), (-0.05, 2e5),
                                     (-0.0625, 0.8), (-0.063, 0.8), (-0.01, 2e4), (-0.01, 2e5), (-0.125, 0.16),
                                     (-0.125, 1.55), (-0.125, 30.0), (-0.125, 2e5)])
def test_no_larger_error_than_fp64(run, dt, size, kind):
    for err in (0.0,) if kind else (0.0, 1.3e-7, -1.3e-7):
        refused, e64, e32, _ = run(dt, size, kind, err)
        assert refused < 20
        assert e32 <= e64, (dt, size, err, e64, e32)


# a passage through the centre multiplies whatever error came before it by a factor of its own orbit, so that the worst
# orbit alone would decide a mean: the median of the orbits' ratios
@pytest.mark.parametrize("kind", [1, 3], ids=["plunging", "at rest"])
@pytest.mark.parametrize("dt,size", [(-0.01, 1.0), (-0.02, 5.0), (-0.05, 1.5), (-0.05, 8.0), (-0.1, 3.0), (-0.125, 3.0),
                                     (-0.125, 8.0)])
def test_through_the_centre(run, dt, size, kind):
    refused, _, _, median = run(dt, size, kind)
    assert refused < 20
    assert median <= 1.0, (dt, size, median)


@pytest.mark.parametrize("dt,size", [(-0.05, 0.05), (-0.01, 0.05), (-0.125, 0.05), (-0.0099, 8.0), (-0.126, 8.0),
                                     (-0.05, 6e5)])
def test_what_is_refused(run, dt, size):
    assert run(dt, size, 2)[0] == 40
