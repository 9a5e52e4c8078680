"""Interfaces of the mixed form under a tolerance that FP32 cannot resolve.

The FP32 iteration for p* may call a root converged only where FP32 can tell
that it is within the caller's tolerance; the others are redone in FP64. FP32
pressures are 2^-24 to 2^-23 of themselves apart: under a tolerance below that
only an iterate that no longer moves counts, and of interfaces between random
states about one in eight keeps moving between neighbouring numbers (13.3 % of
10^6, counted with the solver compiled for the host)."""
import numpy as np
import pytest

from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import FP64, MINMOD, MIXED, OUTFLOW, hydro_params

pytestmark = pytest.mark.gpu

N = 8001


def _step(tol, precision):
    rng = np.random.default_rng(11)
    rho, pr = np.exp(rng.uniform(-1, 1, N)), np.exp(rng.uniform(-1, 1, N))
    vel = 0.5 * rng.uniform(-1, 1, N) * np.sqrt(pr / rho)
    cells = ic.empty_box(1, [N])
    cells[:, 2:-2] = ic.prim_to_cons(rho, [vel], pr, 5.0 / 3.0)
    p = hydro_params(1, limiter=MINMOD, bc=[OUTFLOW] * 2, courant=0.3, tol=tol, precision=precision)
    with gpu.Context(p) as ctx:
        b = ctx.register_box(cells)
        ctx.run(b, [1.0 / N], 1)
        redone = ctx.fallback_count(b)
        ctx.sync_to_host(b)
    return cells[:, 2:-2], redone


@pytest.mark.parametrize("tol", [5e-8, 1e-10, 1e-14])
def test_tolerance_below_fp32_resolution_is_redone_in_fp64(tol):
    state, redone = _step(tol, MIXED)
    assert 0.05 * N < redone < 0.4 * N, redone
    exact, _ = _step(tol, FP64)
    assert np.abs(state - exact).sum() <= 1e-6 * np.abs(exact).sum()


def test_default_tolerance_stays_in_fp32():
    assert _step(1e-6, MIXED)[1] < 0.01 * N
