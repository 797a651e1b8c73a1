"""Ensembles and rollouts where the runtime refuses their cooperative launches:
the same results, launch by launch."""
import fakes
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["full", "segments"])
def test_ensemble(mode):
    fakes.run("""
from opencal_gb300 import ensemble as E, workloads as W
dims = [(48, 56), (33, 40)]
zh = [W.sciddicaT_inputs(r, c, seed=3) for r, c in dims]
def all_of():
    ens = E.Ensemble(dims, [(0.5, 0.001)] * 2, [z for z, _ in zh], [h for _, h in zh], 31)
    ens.set_tape(%r)
    ens.set_graph(False)
    return (ens.forward().cpu().numpy(),) + ens.loss_grad(ens.pack([0.5 * h for _, h in zh]), want_h0_grad=True)
want = all_of()
fake.fake_launches = 0
fake.fake_launch_at = -2
got = all_of()
assert fake.fake_launches >= 3
assert got[0].tobytes() == want[0].tobytes()
assert np.abs(got[1] - want[1]).max() <= 1e-13 * np.abs(want[1]).max()
assert np.abs(got[2] - want[2]).max() <= 1e-12 * np.abs(want[2]).max()
assert got[3].cpu().numpy().tobytes() == want[3].cpu().numpy().tobytes()
""" % mode)


def test_rollout():
    fakes.run("""
import torch
from opencal_gb300 import adjoint, workloads as W
z, h = (torch.from_numpy(a).cuda() for a in W.sciddicaT_inputs(48, 56, seed=3))
def all_of():
    h0 = h.clone().requires_grad_(True)
    r, e = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in (0.5, 0.001))
    hT = adjoint.rollout(z, h0, r, e, 31)
    ((hT - 0.5 * h) ** 2).sum().backward()
    return [x.detach().cpu().numpy() for x in (hT, h0.grad, r.grad, e.grad)]
want = all_of()
fake.fake_launches = 0
fake.fake_launch_at = -2
got = all_of()
assert fake.fake_launches == 2
for k in range(2):
    assert got[k].tobytes() == want[k].tobytes()
for k in range(2, 4):
    assert abs(got[k] - want[k]) <= 1e-12 * abs(want[k])
""")
