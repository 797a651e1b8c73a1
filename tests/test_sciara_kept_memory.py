"""Workspaces that SciaraBatch handles keep between gradients: together at most
a sixteenth of the device's memory, and none after close()."""
import numpy as np
import pytest

from opencal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_bounded_over_all_handles():
    import torch

    import opencal_gb300 as cal
    cal.build()

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    # 48 bytes a cell of fixed arrays and the tape: about 7 GB a handle kept
    rows, cols = 11000, 11000
    z, vents, rates = W.sciara_inputs(64, 64, seed=3, phases=1)
    big = np.full((rows, cols), z.max())
    big[5000:5064, 5000:5064] = z
    vents = [(5000 + x, 5000 + y) for x, y in vents]
    target = np.zeros(rows * cols)
    total = torch.cuda.mem_get_info()[1]
    handles, kept, seen = [], 0, []
    for k in range(4):
        handles.append(cal.SciaraBatch([(big, vents, rates, 600)], list_fraction=1e-3))
        handles[-1].run(2)
        before = used()
        loss, grad, _ = handles[-1].loss_grad(target, 2)
        kept += used() - before
        seen.append((loss.tobytes(), grad[0].tobytes()))
        assert kept <= total / 16 + (256 << 20), k
    assert kept > 5 << 30  # something was kept
    assert np.allclose([np.frombuffer(s[0])[0] for s in seen], np.frombuffer(seen[0][0])[0], rtol=1e-12)
    for h in handles:
        h.close()
