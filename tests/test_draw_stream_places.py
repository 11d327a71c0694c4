"""A place in a pair's random stream (after_gaussians of phygas_gb300/csrc/cuda/pgx_bits.cuh, compiled here as host C++) is
the state that sequential draws reach, also beyond 2^31 Gaussians, which a pair of the most clones whose tries mostly fail
passes."""
import os
import subprocess

CUDA_SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phygas_gb300", "csrc", "cuda")

HARNESS = r"""
#include <cstdio>
#include "pgx_bits.cuh"
using namespace pgx;
int main() {
    const uint64_t seed = 0x123456789abcdef0ull;
    uint64_t s = seed, n = 0;
    int bad = 0;
    // 2^31 + 1,000 Gaussians, two outputs each, one after the other
    for (; n < (1ull << 31) + 1000; n++) {
        if ((n & 0xffffff) == 0 || n + 1000 >= 1ull << 31) bad += after_gaussians(seed, n) != s;
        s += 0x9E3779B97F4A7C15ULL;
        s += 0x9E3779B97F4A7C15ULL;
    }
    bad += after_gaussians(after_gaussians(seed, 1ull << 33), 5) != after_gaussians(seed, (1ull << 33) + 5);
    printf("%d\n", bad);
    return 0;
}
"""


def test_places_beyond_2_31_gaussians(tmp_path):
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", CUDA_SRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.check_output([str(exe)]).split() == [b"0"]
