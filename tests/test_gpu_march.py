"""The last mixed sweep of large boxes (march_kernel) against the tile sweep:
the same operations per cell, so the same bits. A box stepped alone takes the
march from about 156 thousand (column, segment) threads on; in a batch it is
swept in tiles. Where several of a cell's interfaces are redone in FP64 their
contributions are added in any order, in either sweep: near them (two cells a
step) the last bits of the FP64 state may differ, and with them an FP32
rounding of the next step, at most 2^-24 of the state a step."""
import numpy as np
import pytest

from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import (INFLOW, MINMOD, MIXED, OUTFLOW, PERIODIC, REFLECTIVE, SUPERBEE, VAN_ALBADA, VAN_LEER,
                                 hydro_params)

pytestmark = pytest.mark.gpu

DX = 1.0 / 64


def _state(ndim, dims, seed):
    """Waves with a dense block, and a block thin enough for FP64 interfaces."""
    rng = np.random.default_rng(seed)
    x = np.indices(tuple(dims[::-1]))[::-1]
    rho = 1.0 + 0.3 * np.sin(2 * np.pi * sum(x[a] / dims[a] for a in range(ndim)) + rng.uniform())
    vel = [0.3 * np.cos(2 * np.pi * x[(a + 1) % ndim] / dims[(a + 1) % ndim]) for a in range(ndim)]
    pr = 1.0 + 0.2 * rng.uniform(size=rho.shape)
    rho[..., dims[0] // 4:dims[0] // 3] = 4.0
    thin = tuple(slice(n // 2, n // 2 + 3) for n in rho.shape)
    rho[thin] = 1e-7
    pr[thin] = 1e-7
    cells = ic.empty_box(ndim, dims)
    cells[ic.interior(ndim, dims)] = ic.prim_to_cons(rho, vel, pr, 5.0 / 3.0)
    return cells


CASES = [
    (3, [160, 128, 61], [PERIODIC] * 6, SUPERBEE),
    (3, [131, 157, 64], [REFLECTIVE, OUTFLOW, OUTFLOW, REFLECTIVE, OUTFLOW, REFLECTIVE], VAN_LEER),
    (3, [512, 320, 1], [OUTFLOW] * 6, MINMOD),
    (3, [420, 400, 2], [PERIODIC] * 6, VAN_ALBADA),
    (2, [2501, 509], [PERIODIC] * 6, VAN_ALBADA),
    (2, [20001, 65], [REFLECTIVE, REFLECTIVE, REFLECTIVE, OUTFLOW, OUTFLOW, OUTFLOW], SUPERBEE),
    (2, [160003, 8], [OUTFLOW, OUTFLOW, INFLOW, OUTFLOW, OUTFLOW, OUTFLOW], VAN_LEER),
]


@pytest.mark.parametrize("ndim,dims,bc,limiter", CASES)
def test_march_equals_tiles(ndim, dims, bc, limiter):
    p = hydro_params(ndim, bc=bc, limiter=limiter, courant=0.3, precision=MIXED)
    if INFLOW in bc:
        p["inflow"] = [[1.0, 0.0, 0.2, 3.0, 0.0]] * 6
    alone, batched = _state(ndim, dims, 1), _state(ndim, dims, 1)
    with gpu.Context(p) as ctx:
        b = ctx.register_box(alone)
        ctx.run(b, [DX] * ndim, 5)
        redone = ctx.fallback_count(b)
        ctx.sync_to_host(b)
    with gpu.Context(p) as ctx:
        b = ctx.register_box(batched)
        with ctx.batch([b], [[DX] * ndim]) as bt:
            bt.run(5)
        ctx.sync_to_host(b)
    a, t = alone[ic.interior(ndim, dims)], batched[ic.interior(ndim, dims)]
    assert redone > 0 and np.isfinite(a).all()
    near = np.ones(a.shape[1:], dtype=bool)  # the thin block and what it reaches
    for axis, n in enumerate(a.shape[1:]):
        i = np.arange(n).reshape([-1 if k == axis else 1 for k in range(ndim)])
        near &= abs(i - (n // 2 + 1)) <= 2 + 2 * 5
    assert np.array_equal(a[:, ~near], t[:, ~near])
    assert np.max(np.abs(a - t)) <= 5 * 2.0 ** -24 * np.max(np.abs(t))
