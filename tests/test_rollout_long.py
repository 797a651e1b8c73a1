"""A rollout of so many steps on so few cells that its flagged tiles are kept a
segment at a time: forward as the ensemble's, gradient as the segments of an ensemble's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tiles_of_a_segment():
    import torch

    import opencal_gb300 as cal
    from opencal_gb300 import ensemble as E
    cal.build()
    rows, cols, steps = 3, 3, 270_000
    z = np.zeros((rows, cols))
    h = np.zeros((rows, cols))
    h[1, 1] = 2.0
    zt, ht = torch.from_numpy(z).cuda(), torch.from_numpy(h).cuda()

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    h0 = ht.clone().requires_grad_(True)
    r, e = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in (0.2, 0.001))
    before = used()
    hT = cal.adjoint.rollout(zt, h0, r, e, steps)
    # checkpoints, a segment's tiles, four words a step, allocation granules
    assert used() - before <= 8 * rows * cols * 3 * 520 + 24 * steps + (16 << 20)
    ens = E.Ensemble([(rows, cols)], [(0.2, 0.001)], [z], [h], steps)
    assert ens.unpack(ens.forward())[0].tobytes() == hT.detach().cpu().numpy().tobytes()
    target = ens.pack([0.5 * h])
    ((hT - 0.5 * ht) ** 2).sum().backward()
    ens.set_tape("segments")
    loss, grad, gh0 = ens.loss_grad(target, want_h0_grad=True)
    assert ens.unpack(gh0)[0].tobytes() == h0.grad.cpu().numpy().tobytes()
    assert abs(float(r.grad) - grad[0, 0]) <= 1e-12 * abs(grad[0, 0])
    assert abs(float(e.grad) - grad[0, 1]) <= 1e-12 * abs(grad[0, 1])
