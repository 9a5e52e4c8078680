"""Resident runs of any length replay graphs of one and of several steps; the
states and dts must not depend on how a run is cut. Boxes on both sides of
the rules that differ with size: grids within one CTA per SM (launched behind
the kernel before) and larger ones, odd rows (no tensor copies), an extent of
one cell (ghosts filled every step). All boundary types give their ghost cells
from the interior during a run: the ghost cells a run leaves in memory equal
those of the step-by-step calls."""
import numpy as np
import pytest

from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import FP64, INFLOW, MIXED, OUTFLOW, PERIODIC, REFLECTIVE, VAN_LEER, hydro_params

pytestmark = pytest.mark.gpu

BCS = {"periodic": [PERIODIC] * 6, "outflow": [OUTFLOW] * 6, "reflective": [REFLECTIVE] * 6,
       "mixed": [REFLECTIVE, OUTFLOW, INFLOW, OUTFLOW, PERIODIC, PERIODIC]}


def _box(dims, bc, precision, seed=0):
    nd = len(dims)
    rng = np.random.default_rng(seed)
    shp = tuple(dims[::-1])
    vel = [0.2 * rng.uniform(-1, 1, shp) for _ in range(nd)]
    rho, p = 1.0 + 0.3 * rng.uniform(size=shp), 1.0 + 0.3 * rng.uniform(size=shp)
    cells = ic.empty_box(nd, list(dims))
    cells[ic.interior(nd, list(dims))] = ic.prim_to_cons(rho, vel, p, 5.0 / 3.0)
    inflow = np.zeros((6, 5))
    inflow[:, 0], inflow[:, nd + 1] = 1.1, 1.6
    return cells, hydro_params(nd, limiter=VAN_LEER, bc=BCS[bc], courant=0.2, precision=precision, inflow=inflow.tolist())


def _run(cells, p, dx, pieces):
    c = cells.copy()
    dts = []
    with gpu.Context(p) as ctx:
        b = ctx.register_box(c)
        for k in pieces:
            dts.extend(ctx.run(b, dx, k))
        redone = ctx.fallback_count(b)
        ctx.sync_to_host(b)
    return c, np.array(dts), redone


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("dims,bc", [((700,), "mixed"), ((3,), "reflective"), ((40, 33), "mixed"), ((256, 96), "periodic"),
                                     ((24, 20, 9), "mixed"), ((37, 2, 12), "outflow"), ((48, 40, 32), "reflective"),
                                     ((20, 1, 8), "outflow")])
def test_run_does_not_depend_on_its_pieces(dims, bc, precision):
    cells, p = _box(dims, bc, precision)
    dx = [1.0 / max(dims)] * len(dims)
    whole, dts, redone = _run(cells, p, dx, [19])
    assert redone == 0
    for pieces in ([1, 3, 4, 5, 6], [9, 2, 8], [1] * 19):
        c, d, _ = _run(cells, p, dx, pieces)
        assert np.array_equal(d, dts), pieces
        assert np.array_equal(c, whole), pieces


@pytest.mark.parametrize("dims,bc", [((60,), "mixed"), ((40, 33), "mixed"), ((24, 20, 9), "mixed"), ((17, 8, 12), "periodic"),
                                     ((16, 12, 2), "reflective")])
def test_mixed_run_equals_separate_calls(dims, bc):
    cells, p = _box(dims, bc, MIXED, seed=1)
    dx = [1.0 / max(dims)] * len(dims)
    whole, dts, _ = _run(cells, p, dx, [6])
    c = cells.copy()
    with gpu.Context(p) as ctx:
        b = ctx.register_box(c)
        for dt in dts:
            assert ctx.cfl_time_step(b, dx) == dt
            ctx.set_boundaries(b)
            ctx.muscl_hancock_solve(b, dx, dt)
        ctx.sync_to_host(b)
    assert np.array_equal(c, whole)
