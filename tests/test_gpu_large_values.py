"""Mixed boxes whose values come near FP32's largest number (3.4e38): a quotient
by a difference beyond 2^126, for which the fast FP32 division gives 0, must
not flatten a slope. A gas at rest with a ramp and a step in its energy, one
step, against the FP64 path: the first difference of a cell limits its slope
and the second, beyond 2^126, divides it. The FP32 fluxes are within a few
2^-24 of the FP64 ones, a flattened slope is 7 % of the pressure off."""
import numpy as np
import pytest

from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import FP64, LIMITERS, MIXED, OUTFLOW, hydro_params

pytestmark = pytest.mark.gpu

N = 40


def _step(precision, limiter, omega, ndim, mirrored):
    e = np.full(N, 1.0e38)
    e[20:] = 1.2e38
    e[21:] = 2.2e38
    if mirrored:
        e = e[::-1]
    dims = [N] + [5] * (ndim - 1)
    shp = tuple(dims[::-1])
    cells = ic.empty_box(ndim, dims)
    inner = ic.interior(ndim, dims)
    w = np.zeros((ndim + 2,) + shp)
    w[0], w[-1] = 1.0e37, np.broadcast_to(e, shp)
    cells[inner] = w
    p = hydro_params(ndim, limiter=limiter, omega=omega, bc=[OUTFLOW] * 6, courant=0.3, precision=precision)
    with gpu.Context(p) as ctx:
        b = ctx.register_box(cells)
        dt = ctx.run(b, [1.0 / N] * ndim, 1)[0]
        ctx.sync_to_host(b)
    return cells[inner], dt


@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("mirrored", [False, True])
@pytest.mark.parametrize("omega", [0.0, 0.25])
@pytest.mark.parametrize("limiter", sorted(LIMITERS))
def test_step_beyond_2_126(limiter, omega, mirrored, ndim):
    a, dta = _step(FP64, LIMITERS[limiter], omega, ndim, mirrored)
    b, dtb = _step(MIXED, LIMITERS[limiter], omega, ndim, mirrored)
    assert np.isfinite(a).all() and abs(dta - dtb) <= 1e-6 * dta
    for c in (0, 1, ndim + 1):
        assert np.max(np.abs(a[c] - b[c])) <= 1e-5 * np.max(np.abs(a[c])), c
