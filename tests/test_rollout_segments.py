"""The sqrt(T) form of a rollout's backward, which otherwise only runs where a
whole rollout's tape does not fit in memory: dL/dh0, dL/dr and dL/deps bit for
bit as with the whole tape (the same additions in the same order)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# steps: one, whole segments, a last segment of one step, and of some
@pytest.mark.parametrize("steps", [0, 1, 2, 16, 17, 50])
@pytest.mark.parametrize("rows,cols,toroidal", [(1, 1, 1), (40, 31, 0), (49, 65, 1)])
def test_segments_equal_the_whole_tape(steps, rows, cols, toroidal):
    import torch

    import opencal_gb300 as cal
    cal.build()
    lib = cal.adjoint._lib()
    rng = np.random.default_rng(rows * 100 + cols)
    z = np.floor(rng.random((rows, cols)) * 2048) / 1024 + 0.125 * np.arange(rows)[:, None]
    h = np.where(rng.random((rows, cols)) < 0.3, np.floor(rng.random((rows, cols)) * 8192) / 1024, 0.0)
    z, h = torch.from_numpy(z).cuda(), torch.from_numpy(h).cuda()
    got = []
    for mode in (1, 2):
        hd = lib.cal_sdt_adj_create(rows, cols, steps, toroidal)
        assert hd and lib.cal_sdt_adj_set_tape(hd, mode) == 0 and lib.cal_sdt_adj_set_tape(hd, 3) == 1
        try:
            for scale in (1.0, 0.25):  # two rollouts of one workspace, two backwards each
                h0, hT = scale * h, torch.empty_like(h)
                st = torch.cuda.current_stream().cuda_stream
                assert lib.cal_sdt_adj_forward(hd, z.data_ptr(), h0.data_ptr(), 0.5, 0.001, hT.data_ptr(), st) == 0
                for seed in (2.0 * hT, torch.ones_like(hT)):
                    g, gr, ge = torch.empty_like(h), C.c_double(), C.c_double()
                    assert lib.cal_sdt_adj_backward(hd, seed.data_ptr(), g.data_ptr(), C.byref(gr), C.byref(ge),
                                                    st) == 0
                    got.append((mode, hT.cpu().numpy().tobytes(), g.cpu().numpy().tobytes(), gr.value, ge.value))
        finally:
            lib.cal_sdt_adj_destroy(hd)
    for k in range(4):
        assert got[k][1:] == got[4 + k][1:]
