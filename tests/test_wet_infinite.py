"""Parameter gradients that overflow: infinite where the sum of the cells'
parts is, and the others of the ensemble are what they are alone."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2])
def test_infinite_sum(mode):
    import torch

    import opencal_gb300 as cal
    cal.build()
    lib = cal.adjoint._lib()
    rows = cols = 40
    z, h = torch.zeros(rows, cols, dtype=torch.float64), torch.zeros(rows, cols, dtype=torch.float64)
    for i in range(3, 38, 7):  # wet cells that do not share a neighbour
        for j in range(3, 38, 7):
            h[i, j] = 1.0
    z += h  # the initialisation takes it off again
    gT = torch.ones_like(h)
    gT[10, 10] = -1.7e308  # lambda of a neighbour minus this: infinite
    gT[9, 10] = 1.7e308
    z, h, gT = z.cuda(), h.cuda(), gT.cuda()
    hd = lib.cal_sdt_adj_create(rows, cols, 1, 0)
    assert lib.cal_sdt_adj_set_tape(hd, mode) == 0
    try:
        st = torch.cuda.current_stream().cuda_stream
        hT, g, gr, ge = torch.empty_like(h), torch.empty_like(h), C.c_double(), C.c_double()
        assert lib.cal_sdt_adj_forward(hd, z.data_ptr(), h.data_ptr(), 0.5, 0.001, hT.data_ptr(), st) == 0
        assert lib.cal_sdt_adj_backward(hd, gT.data_ptr(), g.data_ptr(), C.byref(gr), C.byref(ge), st) == 0
    finally:
        lib.cal_sdt_adj_destroy(hd)
    assert gr.value == np.inf


def test_ensemble_neighbours_stay_finite():
    import opencal_gb300 as cal
    from opencal_gb300 import ensemble as E
    from opencal_gb300 import workloads as W
    cal.build()
    dims = [(48, 56), (40, 40), (33, 41)]
    zh = [W.sciddicaT_inputs(r, c, seed=3) for r, c in dims]
    ens = E.Ensemble(dims, [(0.5, 0.001)] * 3, [z for z, _ in zh], [h for _, h in zh], 20)
    target = [0.5 * h for _, h in zh]
    want = ens.loss_grad(ens.pack(target))[1]
    target[1] = target[1] + 1e308 * np.where((np.add.outer(np.arange(40), np.arange(40)) % 2) == 0, 1.0, -1.0)
    got = ens.loss_grad(ens.pack(target))[1]
    assert got[0].tobytes() == want[0].tobytes() and got[2].tobytes() == want[2].tobytes()
    assert not np.isfinite(got[1]).all()
