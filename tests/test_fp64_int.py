"""The integer FP64 division, square root, comparisons and power-of-two
scaling of the FP64 kernels (fp64_int.h) against the host's IEEE operations,
bit for bit: any operands, ordinary magnitudes, short significands, both
sides of a power of two, special values, numerators and squares next to a
midpoint of the result; with the FP32 seeds of the reciprocal and the root
exact and off by 1.5e-7 to either side (the hardware's are within 1.2e-7)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fp64_int") / "check")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", os.path.join(HERE, "fp64_int_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed_error", ["0", "1.5e-7", "-1.5e-7"])
@pytest.mark.parametrize("kind", range(6))
def test_equals_ieee(program, kind, seed_error):
    r = subprocess.run([program, str(kind), "500000", seed_error], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
