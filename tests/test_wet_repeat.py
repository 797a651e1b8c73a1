"""Gradients of rollouts and ensembles repeat bit for bit: nothing in them
depends on the order in which the lists of wet cells were appended."""
import numpy as np
import pytest

from opencal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,steps", [(40, 33, 1), (97, 80, 60), (400, 300, 150)])
@pytest.mark.parametrize("toroidal", [False, True])
def test_rollout(rows, cols, steps, toroidal):
    import torch

    import opencal_gb300 as cal
    cal.build()
    z, h = (torch.from_numpy(a).cuda() for a in W.sciddicaT_inputs(rows, cols, seed=rows))
    seen = set()
    for _ in range(6):
        h0 = h.clone().requires_grad_(True)
        r, e = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in (0.5, 0.001))
        ((cal.adjoint.rollout(z, h0, r, e, steps, toroidal) - 0.5 * h) ** 2).sum().backward()
        seen.add((float(r.grad), float(e.grad), h0.grad.cpu().numpy().tobytes()))
    assert len(seen) == 1 and list(seen)[0][0] != 0.0


@pytest.mark.parametrize("mode", ["full", "segments"])
def test_ensemble(mode):
    import opencal_gb300 as cal
    from opencal_gb300 import ensemble as E
    cal.build()
    dims = [(1, 1), (130, 97), (64, 300), (33, 31), (200, 210)]
    zh = [W.sciddicaT_inputs(r, c, seed=7) if r > 1 else (np.zeros((1, 1)), np.ones((1, 1))) for r, c in dims]
    ens = E.Ensemble(dims, [(0.5, 0.001)] * len(dims), [z for z, _ in zh], [h for _, h in zh], 60)
    ens.set_tape(mode)
    target = ens.pack([0.5 * h for _, h in zh])
    seen = set()
    for k in range(6):
        ens.set_graph(k % 2 == 0)
        seen.add(ens.loss_grad(target)[1].tobytes())
    assert len(seen) == 1
