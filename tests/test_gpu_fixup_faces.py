"""FP64 redo of interfaces at the box's faces: a resident run and a batch run
take the ghost cells of their stencils from the interior (all boundary types),
the separate calls from memory. With one iteration allowed nearly every
interface between differing states is redone, those at and next to each face
among them.

A redo's two contributions are added atomically, in any order: an FP64
rounding, which at most flips an FP32 rounding of the next step's mirror
(2^-24 of the state). A step at these Courant numbers passes a difference on
to a cell's neighbours with a weight below 3 in all, so after 6 steps the runs
may differ by (3^6 - 1)/2 2^-24 < 3e-5 of the largest value; a ghost cell from
the wrong place or with the wrong sign changes a flux by some percent."""
import numpy as np
import pytest

from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import INFLOW, MIXED, OUTFLOW, PERIODIC, REFLECTIVE, VAN_LEER, hydro_params

pytestmark = pytest.mark.gpu

TOL = 3e-5
BCS = {"reflective": [REFLECTIVE] * 6, "outflow": [OUTFLOW] * 6, "periodic": [PERIODIC] * 6, "inflow": [INFLOW] * 6,
       "mixed": [REFLECTIVE, INFLOW, OUTFLOW, REFLECTIVE, INFLOW, OUTFLOW]}
DIMS = [(9,), (70,), (2,), (12, 7), (37, 33), (8, 6, 5), (16, 12, 2), (17, 12, 6)]


def _box(dims, bc):
    nd = len(dims)
    rng = np.random.default_rng(5)
    shp = tuple(dims[::-1])
    vel = [0.3 * rng.uniform(-1, 1, shp) for _ in range(nd)]
    rho, pr = 1.0 + 0.5 * rng.uniform(size=shp), 1.0 + 0.5 * rng.uniform(size=shp)
    cells = ic.empty_box(nd, list(dims))
    cells[ic.interior(nd, list(dims))] = ic.prim_to_cons(rho, vel, pr, 5.0 / 3.0)
    inflow = np.zeros((6, 5))
    inflow[:, 0], inflow[:, 1:1 + nd], inflow[:, nd + 1] = 1.2, 0.1, 2.0
    return cells, hydro_params(nd, limiter=VAN_LEER, bc=BCS[bc], courant=0.2, n_iter=1, precision=MIXED,
                               inflow=inflow.tolist())


def _separate(p, cells, dx, steps):
    c, dts = cells.copy(), []
    with gpu.Context(p) as ctx:
        b = ctx.register_box(c)
        for _ in range(steps):
            dts.append(ctx.cfl_time_step(b, dx))
            ctx.set_boundaries(b)
            ctx.muscl_hancock_solve(b, dx, dts[-1])
        redone = ctx.fallback_count(b)
        ctx.sync_to_host(b)
    return c, np.array(dts), redone


@pytest.mark.parametrize("bc", sorted(BCS))
@pytest.mark.parametrize("dims", DIMS)
def test_redone_interfaces_at_the_faces(dims, bc):
    nd, steps = len(dims), 6
    cells, p = _box(dims, bc)
    dx = [1.0 / 16] * nd
    ref, dts, redone = _separate(p, cells, dx, steps)
    inner = ic.interior(nd, list(dims))
    scale = np.max(np.abs(ref[inner]))
    interior_faces = sum(np.prod(dims) // dims[a] * (dims[a] - 1) for a in range(nd))
    assert np.isfinite(ref[inner]).all() and redone > 0.8 * steps * interior_faces
    for pieces in ([6], [1, 5], [3, 3], [1] * 6):
        for how in ("run", "batch"):
            c, got = cells.copy(), []
            with gpu.Context(p) as ctx:
                b = ctx.register_box(c)
                if how == "run":
                    for k in pieces:
                        got.extend(ctx.run(b, dx, k))
                else:
                    with ctx.batch([b], [dx]) as bt:
                        for k in pieces:
                            bt.run(k)
                again = ctx.fallback_count(b) if how == "run" else None
                ctx.sync_to_host(b)
            assert np.max(np.abs(c[inner] - ref[inner])) <= TOL * scale, (pieces, how)
            if how == "run":
                assert np.allclose(got, dts, rtol=TOL, atol=0.0)
                assert abs(again - redone) <= 0.02 * redone, pieces
