"""Device memory of live rollouts: what one holds between its forward and its
backward, and after it, is bounded by what sqrt(T) checkpointing holds (or a
128th of the free memory, where that is more), and the gradients do not
depend on whether the tape fitted."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _used(torch):
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("rows,cols,steps,wet", [(512, 480, 900, 0.02), (1024, 1024, 400, 0.01), (600, 500, 100, 0.9),
                                                 (2048, 1900, 300, 0.02)])
def test_bounded_by_checkpointing(rows, cols, steps, wet):
    import torch

    import opencal_gb300 as cal
    cal.build()
    rng = np.random.default_rng(rows)
    z = torch.from_numpy(np.floor(rng.random((rows, cols)) * 2048) / 1024).cuda()
    h = torch.from_numpy(np.where(rng.random((rows, cols)) < wet, 1.0, 0.0)).cuda()
    K = math.ceil(math.sqrt(steps))
    n = rows * cols
    # the tape, 24 fields of the workspace, the tiles of every step, allocation granules
    tape = max(8 * n * (K + math.ceil(steps / K) + 1), torch.cuda.mem_get_info()[0] // 128)
    bound = tape + 8 * n * 24 + 4 * (n // 256 + rows + cols) * (steps + 1) + (64 << 20)

    def rollout():
        h0 = h.clone().requires_grad_(True)
        r, e = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in (0.4, 0.001))
        return h0, r, e, cal.adjoint.rollout(z, h0, r, e, steps)

    warm = rollout()
    del warm
    torch.cuda.empty_cache()
    before = _used(torch)
    h0, r, e, hT = rollout()
    assert _used(torch) - before <= bound
    loss = (hT ** 2).sum()
    first = torch.autograd.grad(loss, (h0, r, e), retain_graph=True)
    torch.cuda.empty_cache()
    assert _used(torch) - before <= bound + 8 * 8 * n
    again = torch.autograd.grad(loss, (h0, r, e), retain_graph=True)
    for a, b in zip(first, again):
        assert a.cpu().numpy().tobytes() == b.cpu().numpy().tobytes()
