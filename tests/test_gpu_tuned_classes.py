"""No sweep runs with a tile shape that was timed for another kernel: a 2-D
batch sweeps in tiles where a resident run marches along the last axis and has
classes of its own, a box whose last sweep marches is not of the class of one
whose sweep does not, and the solve with overlapped write-back, which neither
fuses x and y nor marches, takes the size rule's shapes."""
import numpy as np
import pytest

from rhyme_gb300 import gpu, ic
from rhyme_gb300.params import MIXED, PERIODIC, hydro_params

pytestmark = pytest.mark.gpu


def _box(dims):
    nd, shp = len(dims), tuple(dims[::-1])
    rng = np.random.default_rng(3)
    cells = ic.empty_box(nd, list(dims))
    cells[ic.interior(nd, list(dims))] = ic.prim_to_cons(1.0 + 0.2 * rng.uniform(size=shp),
                                                         [0.1 * rng.uniform(size=shp) for _ in range(nd)],
                                                         1.0 + 0.2 * rng.uniform(size=shp), 5.0 / 3.0)
    return cells, [1.0 / max(dims)] * nd


def _params(nd):
    return hydro_params(nd, bc=[PERIODIC] * 6, courant=0.3, precision=MIXED)


def test_write_back_solve_takes_no_shape_timed_for_another_kernel():
    cells, dx = _box((160, 128, 64))  # a resident run marches with 8-cell segments
    host = cells.copy()
    with gpu.Context(_params(3)) as ctx:
        b = ctx.register_box(host)
        ctx.set_host_writeback(b, True)
        dt = ctx.cfl_time_step(b, dx)
        ctx.set_boundaries(b)
        ctx.muscl_hancock_solve(b, dx, dt)
        ctx.sync_to_host(b)
        assert ctx.tuned_classes() == 0
        ctx.sweep_plan(b, dx)
        assert ctx.tuned_classes() == 1  # z alone: x and y are one kernel
    with gpu.Context(_params(3)) as ctx:
        b = ctx.register_box(cells)
        assert ctx.run(b, dx, 1)[0] == dt
        ctx.sync_to_host(b)
    inner = ic.interior(3, [160, 128, 64])
    assert np.array_equal(host[inner], cells[inner])


def test_marching_box_has_its_own_class():
    with gpu.Context(_params(3)) as ctx:
        for k, dims in enumerate([(160, 16, 64), (160, 128, 64), (160, 100, 64)]):
            cells, dx = _box(dims)
            ctx.sweep_plan(ctx.register_box(cells), dx)
            assert ctx.tuned_classes() == (1, 2, 2)[k]


def test_batch_of_a_large_2d_box_has_its_own_shapes():
    cells, dx = _box((1100, 1200))
    with gpu.Context(_params(2)) as ctx:
        b = ctx.register_box(cells)
        ctx.sweep_plan(b, dx)
        assert ctx.tuned_classes() == 2
        with ctx.batch([b], [dx]) as bt:
            assert ctx.tuned_classes() == 3  # y in tiles; x is the same kernel
            bt.run(2)


@pytest.mark.parametrize("nd", [1, 2])
def test_batch_with_tuned_shapes_equals_boxes_alone(nd):
    """Boxes of several size classes, each with the shapes of its class."""
    all_dims = {1: [(40,), (300,), (1500,)], 2: [(12, 90), (64, 16), (40, 130), (200, 40)]}[nd]
    boxes = [_box(d) for d in all_dims]
    alone = []
    for cells, dx in boxes:
        c = cells.copy()
        with gpu.Context(_params(nd)) as ctx:
            b = ctx.register_box(c)
            ctx.run(b, dx, 5)
            ctx.sync_to_host(b)
        alone.append(c)
    with gpu.Context(_params(nd)) as ctx:
        hs = [ctx.register_box(cells) for cells, _ in boxes]
        with ctx.batch(hs, [dx for _, dx in boxes]) as bt:
            assert ctx.tuned_classes() >= nd * 2
            bt.run(5)
        for h in hs:
            ctx.sync_to_host(h)
    for (cells, _), a in zip(boxes, alone):
        assert np.array_equal(cells, a)
