"""A rollout whose tape holds a part of its steps: the sweep goes back over what
the tape holds and runs the steps before it again, as often as it takes.  Every
gradient bit for bit as with the whole tape (the same additions in the same
order), two forwards of a workspace and two backwards each."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the largest fraction still misses an entry; 0.3 and less cost more than a
# forward, and a tape that fits is allocated for the sweep instead
@pytest.mark.parametrize("fraction", [1.0, 0.95, 0.8, 0.6, 0.45, 0.3, 0.1, 0.0])
@pytest.mark.parametrize("rows,cols,steps,toroidal", [(40, 31, 50, 0), (49, 65, 17, 1), (30, 30, 2, 0), (96, 80, 200, 0)])
def test_same_gradients(fraction, rows, cols, steps, toroidal):
    import torch

    import opencal_gb300 as cal
    cal.build()
    lib = cal.adjoint._lib()
    rng = np.random.default_rng(rows * 100 + cols)
    z = np.floor(rng.random((rows, cols)) * 2048) / 1024 + 0.125 * np.arange(rows)[:, None]
    h = np.where(rng.random((rows, cols)) < 0.3, np.floor(rng.random((rows, cols)) * 8192) / 1024, 0.0)
    h[rows // 2:] = 0.0  # the flow grows: later steps have more entries
    z, h = torch.from_numpy(z).cuda(), torch.from_numpy(h).cuda()
    # entries of the whole rollout: the wet cells of every step and the cells that dried
    need = 0
    wet = h > 0.001
    for t in range(steps):
        now = cal.adjoint.rollout(z, h, 0.5, 0.001, t, bool(toroidal)) > 0.001
        need += int(now.sum()) + (int((wet & ~now).sum()) if t else 0)
        wet = now
    got = []
    for limit in (0, max(1, int(fraction * (need - 1)))):
        hd = lib.cal_sdt_adj_create(rows, cols, steps, toroidal)
        assert hd and lib.cal_sdt_adj_set_tape_limit(hd, limit) == 0 and lib.cal_sdt_adj_set_tape_limit(hd, -1) == 1
        try:
            for scale in (1.0, 0.25):
                h0, hT = scale * h, torch.empty_like(h)
                st = torch.cuda.current_stream().cuda_stream
                assert lib.cal_sdt_adj_forward(hd, z.data_ptr(), h0.data_ptr(), 0.5, 0.001, hT.data_ptr(), st) == 0
                for seed in (2.0 * hT, torch.ones_like(hT)):
                    g, gr, ge = torch.empty_like(h), C.c_double(), C.c_double()
                    assert lib.cal_sdt_adj_backward(hd, seed.data_ptr(), g.data_ptr(), C.byref(gr), C.byref(ge),
                                                    st) == 0
                    got.append((hT.cpu().numpy().tobytes(), g.cpu().numpy().tobytes(), gr.value, ge.value))
        finally:
            lib.cal_sdt_adj_destroy(hd)
    for k in range(4):
        assert got[k] == got[4 + k]
