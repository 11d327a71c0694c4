"""The float-pair force (phygas_gb300/csrc/cuda/pgx_orbit32.cuh) at the halo's cut-off, where the force has a kink: positions
within a few 10^-6 kpc of it, on both sides, take their own side's formula.  Against 113-bit arithmetic."""
import subprocess

import pytest

from tests.test_orbit32 import CUDA_SRC, HARNESS, harness      # noqa: F401  (harness: skips where 113 bits are missing)

MAIN = r"""
int main() {
    std::vector<Halo32> halo(kHalo32N);
    for (int n = 0; n < kHalo32N; n++) halo[n] = halo32_entry(n, Model::a, kInvA);
    auto table = [&](int n) { return halo[n]; };
    OrbitScale s;
    if (!orbit32_scale(200.0, 0.05, s)) return 2;
    const Force32 K = force32_constants<Model>(0.05, s);
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    double worst = 0;
    for (int k = 0; k < 4000; k++) {
        double d[3] = {U(g), U(g), U(g)};
        const double n = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]), r = 100.0 + 1e-5 * U(g);
        int64_t x[3];
        Q p[3], a[3];
        F2 f[3];
        for (int c = 0; c < 3; c++) {
            x[c] = f64_to_i64(ldexp(d[c] / n * r, 55));
            p[c] = (Q)x[c] * (Q)ldexp(1.0, -55);
            f[c] = fixed_to_f2(x[c], s.c);
        }
        accel<Q>(p, a);
        const Acc32 A = force32<Model>(K, table, f[0], f[1], f[2]);
        const F2 got[3] = {A.x, A.y, A.z};
        double e2 = 0, a2 = 0;
        for (int c = 0; c < 3; c++) {
            const Q want = a[c] * (Q)(0.05 * 0.05) * (Q)ldexp(1.0, 37);
            const double e = (double)((Q)got[c].h + (Q)got[c].l - want);
            e2 += e * e;
            a2 += (double)(want * want);
        }
        worst = fmax(worst, sqrt(e2 / a2));
    }
    printf("%.6e\n", worst);
    return 0;
}
"""


def test_each_side_of_the_cut_off_takes_its_own_formula(harness, tmp_path):      # noqa: F811
    src, exe = tmp_path / "k.cpp", tmp_path / "k"
    src.write_text(HARNESS[:HARNESS.index("int main(")] + MAIN)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-I", CUDA_SRC, str(src), "-o", str(exe),
                    "-lquadmath"], check=True)
    # some sixteen operations in a chain, each within 2^-47: 2^-43 at worst
    assert float(subprocess.check_output([str(exe)])) < 2.0 ** -43
