"""The model's constants that the float-pair orbit's CPU tests restate (tests/test_orbit32.py) are those of the device's
model (phygas_gb300/csrc/cuda/pgx_internal.cuh, pgx_force.cuh)."""
import os
import re

from tests.test_orbit32 import CUDA_SRC, HARNESS


def constants(text, names=None):
    """The `constexpr double name = expression` values of a source, in order."""
    out = dict(names or {})
    text = re.sub(r"//[^\n]*", "", text)
    for decl in re.findall(r"constexpr double ([^;]+);", text):
        for part in re.split(r",\s*(?=k\w+\s*=)", decl):
            name, expr = (x.strip() for x in part.split("=", 1))
            try:
                out[name] = eval(expr, {}, out)
            except (NameError, SyntaxError):
                pass
    return out


def test_the_restated_constants():
    with open(os.path.join(CUDA_SRC, "pgx_internal.cuh")) as f:
        device = constants(f.read())
    host = constants(HARNESS)
    pairs = {"kKms": "kKms", "kG": "kG", "kBulge": "kBulgeGM", "kB2": "kBulgeB2", "kDisk": "kDiskGM", "kA": "kDiskA",
             "kD2": "kDiskB2", "kHalo": "kHaloGM", "kInvA": "kHaloInvA", "kPow": "kHaloG1"}
    for h, d in pairs.items():
        assert host[h] == device[d], (h, host[h], device[d])
    assert "split3(%r)" % device["kHaloFar"] in HARNESS
    assert float(re.search(r"cut2 = (\w+)f", HARNESS).group(1)) == device["kHaloCut"] ** 2
