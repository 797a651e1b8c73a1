"""cal_sdt_adj_forward captured into a CUDA graph: each replay runs the rollout
from what h0 holds then, and a backward after it is that rollout's."""
import ctypes as C

import numpy as np
import pytest

from opencal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 40])
@pytest.mark.parametrize("warm", [False, True])
def test_captured_forward(steps, warm):
    import torch

    import opencal_gb300 as cal
    cal.build()
    lib = cal.adjoint._lib()
    rows, cols = 70, 61
    z, h = (torch.from_numpy(a).cuda() for a in W.sciddicaT_inputs(rows, cols, seed=9))
    hd = lib.cal_sdt_adj_create(rows, cols, steps, 0)
    h0, hT, g = h.clone(), torch.empty_like(h), torch.empty_like(h)

    def forward():
        st = torch.cuda.current_stream().cuda_stream
        return lib.cal_sdt_adj_forward(hd, z.data_ptr(), h0.data_ptr(), 0.5, 0.001, hT.data_ptr(), st)

    try:
        if warm:
            assert forward() == 0
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            assert forward() == 0
        for scale in (1.0, 0.5, 1.0):
            h0.copy_(h * scale)
            graph.replay()
            torch.cuda.synchronize()
            x = (h * scale).requires_grad_(True)
            r, e = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in (0.5, 0.001))
            ref = cal.adjoint.rollout(z, x, r, e, steps)
            assert hT.cpu().numpy().tobytes() == ref.detach().cpu().numpy().tobytes()
            (ref ** 2).sum().backward()
            gr, ge = C.c_double(), C.c_double()
            seed = 2.0 * hT
            torch.cuda.synchronize()
            assert lib.cal_sdt_adj_backward(hd, seed.data_ptr(), g.data_ptr(), C.byref(gr), C.byref(ge), None) == 0
            assert g.cpu().numpy().tobytes() == x.grad.cpu().numpy().tobytes()
            assert np.float64(gr.value) == float(r.grad) and np.float64(ge.value) == float(e.grad)
    finally:
        lib.cal_sdt_adj_destroy(hd)


def test_captured_ensemble_forward():
    import torch

    import opencal_gb300 as cal
    from opencal_gb300 import ensemble as E
    cal.build()
    dims = [(40, 33), (70, 61)]
    zh = [W.sciddicaT_inputs(r, c, seed=9) for r, c in dims]
    ens, ref = (E.Ensemble(dims, [(0.5, 0.001)] * 2, [z for z, _ in zh], [h for _, h in zh], 25) for _ in range(2))
    hT = torch.empty(ens.cells, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(ens._lib.cal_sdt_batch_stream(ens.handle))):
        assert ens._lib.cal_sdt_batch_forward(ens.handle, C.c_void_p(hT.data_ptr())) == 0
    for r in (0.5, 0.3):
        for e in (ens, ref):
            e.set_params([(r, 0.001)] * 2)
        want = ref.forward()
        assert ens.forward().cpu().numpy().tobytes() == want.cpu().numpy().tobytes()
        graph.replay()
        torch.cuda.synchronize()
        assert hT.cpu().numpy().tobytes() == want.cpu().numpy().tobytes()
