"""The FP64 wave functions' quotient by twice a number whose reciprocal is
known (fp64_int.h) against the host's IEEE quotient, bit for bit: ordinary
divisors, subnormal ones, those whose double is the first normal number or
overflows, any."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("div_by_twice") / "check")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", os.path.join(HERE, "div_by_twice_check.cpp"), "-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("seed_error", ["0", "1.5e-7", "-1.5e-7"])
@pytest.mark.parametrize("kind", range(4))
def test_equals_ieee(program, kind, seed_error):
    r = subprocess.run([program, str(kind), "500000", seed_error], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
