"""What a server holds of the GPU's memory between requests is bounded by its
HBM budget, whatever the dimensionalities of the requests it has served: at
most a quarter of the budget stays with it when nothing is active."""
import numpy as np
import pytest

from rhyme_gb300 import drawing, gpu, ic
from rhyme_gb300.params import FP64, OUTFLOW, hydro_params

pytestmark = pytest.mark.gpu

BUDGET = 2 << 30


def _serve(srv, dims):
    nd = len(dims)
    cells = ic.empty_box(nd, list(dims))
    shapes = drawing.spheres_3d(n=min(dims), nspheres=1, seed=1) if nd == 3 else None
    if shapes is None:
        cells[ic.interior(nd, list(dims))] = ic.prim_to_cons(np.ones(dims[::-1]), [np.zeros(dims[::-1])] * nd,
                                                             np.ones(dims[::-1]), 5.0 / 3.0)
    rid = srv.submit(cells, 1, [1.0 / max(dims)] * nd, 1, [OUTFLOW] * 6, shapes=shapes)
    for _ in range(200000):
        if srv.tick() == (0, 0, 0):
            break
    assert srv.request(rid)[0] == gpu.REQ_DONE


def test_idle_server_keeps_a_quarter_of_its_budget():
    torch = pytest.importorskip("torch")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    with gpu.Server(hydro_params(3, precision=FP64), (0.8, 0.5, 0.3), BUDGET, 8) as srv:
        for dims in ((64,), (16, 16), (8, 8, 8)):  # every kernel loaded
            _serve(srv, dims)
        before = free()
        for dims in ((4000000,), (1400, 1400), (104, 104, 104)):  # 0.5 GB each
            _serve(srv, dims)
        held = before - free()
    assert held <= BUDGET // 4 + (64 << 20), held / 2 ** 20
