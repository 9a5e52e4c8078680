"""The status word of mixed boxes tells of states that exist: what a step's
last sweep leaves before the FP64 fix-up has added the fluxes of the redone
interfaces is none; the state after it is one, also when no step follows."""
import numpy as np
import pytest

import oracle
from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import MINMOD, MIXED, OUTFLOW, VAN_LEER, hydro_params

pytestmark = pytest.mark.gpu

G = 5.0 / 3.0


def _box(ndim, u, p, rows=6):
    dims = [len(u)] + [rows] * (ndim - 1)
    shp = tuple(dims[::-1])
    cells = ic.empty_box(ndim, dims)
    vel = [np.broadcast_to(u, shp)] + [np.zeros(shp)] * (ndim - 1)
    cells[ic.interior(ndim, dims)] = ic.prim_to_cons(np.ones(shp), vel, np.broadcast_to(p, shp), G)
    return cells, [1.0 / len(u)] * ndim


def _pressure(w):
    return (G - 1.0) * (w[-1] - 0.5 * np.sum(w[1:-1] ** 2, axis=0) / w[0])


def _stepper(ctx, box, dx, how):
    """run(steps) of the box alone or of a batch of it."""
    if how == "run":
        return lambda k: ctx.run(box, dx, k)
    return ctx.batch([box], [dx]).run


@pytest.mark.parametrize("how", ["run", "batch"])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_physical_state_after_redone_interfaces(ndim, how):
    """A cold fast flow with one pressure jump, whose interface two iterations
    do not solve: without that interface's flux the cell behind it would have
    a pressure of -0.37 (+0.6 with it)."""
    u, p = np.full(32, 20.0), np.full(32, 0.6)
    u[12:] += 5.0
    u[13:] += 4.0
    p[:12] *= 3.0
    cells, dx = _box(ndim, u, p)
    q = hydro_params(ndim, limiter=VAN_LEER, bc=[OUTFLOW] * 6, courant=0.4, n_iter=2, precision=MIXED)
    ref = cells.copy()
    oracle.run(dict(q, precision=0), ref, dx, 1)
    inner = ic.interior(ndim, [32] + [6] * (ndim - 1))
    assert _pressure(ref[inner]).min() > 0.5
    with gpu.Context(q) as ctx:
        b = ctx.register_box(cells)
        step = _stepper(ctx, b, dx, how)
        step(1)
        if how == "run":  # (a batch keeps its own count)
            assert ctx.fallback_count(b) > 0
        assert ctx.box_status(b) == 0
        ctx.sync_to_host(b)
        assert _pressure(cells[inner]).min() > 0.5
        step(1)
        assert ctx.box_status(b) == 0


@pytest.mark.parametrize("how", ["run", "batch"])
def test_unphysical_state_is_reported_after_its_step(how):
    """Two receding states at a Courant number at which the scheme itself
    reaches a negative pressure within some tens of steps."""
    u, p = np.where(np.arange(256) < 128, -3.0, 3.0), np.full(256, 0.05)
    cells, dx = _box(1, u, p)
    q = hydro_params(1, limiter=MINMOD, bc=[OUTFLOW] * 2, vac_rho=1e-8, vac_p=1e-10, courant=0.5, precision=MIXED)
    seen = set()
    with gpu.Context(q) as ctx:
        b = ctx.register_box(cells)
        step = _stepper(ctx, b, dx, how)
        before = False
        for _ in range(80):
            step(1)
            status = ctx.box_status(b)
            ctx.sync_to_host(b)
            w = cells[:, 2:-2]
            if not np.isfinite(w).all():
                break
            pr = _pressure(w)
            bad = bool((w[0] <= 0).any() or (pr < -1e-4).any())
            fine = bool((w[0] > 1e-7).all() and (pr > 1e-4).all())
            if bad:
                assert status & 1
                seen.add("bad")
            elif fine and not before:
                assert status == 0
                seen.add("fine")
            before = not fine
    assert seen == {"bad", "fine"}, seen
