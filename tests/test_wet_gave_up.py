"""The runs after one whose grid barrier gave up (the abandoned run's flows are
still in memory): ensembles and rollouts answer as if it had not been."""
import fakes
import pytest

pytestmark = pytest.mark.gpu

ENSEMBLE = """
from opencal_gb300 import ensemble as E, workloads as W
dims = [(48, 56), (33, 40)]
zh = [W.sciddicaT_inputs(r, c, seed=3) for r, c in dims]
ens = E.Ensemble(dims, [(0.5, 0.001)] * 2, [z for z, _ in zh], [h for _, h in zh], 31)
want = ens.forward().cpu().numpy()
target = ens.pack([0.5 * h for _, h in zh])
loss, grad, gh0 = ens.loss_grad(target, want_h0_grad=True)
fake.fake_cut_at = 0
assert np.isnan(ens.forward().cpu().numpy()).all()
"""


def test_ensemble_forward_after_one_that_gave_up():
    fakes.run(ENSEMBLE + """
try:
    ens.active_tiles()
    raise SystemExit("no error")
except Exception as e:
    assert "active_tiles" in str(e)
assert ens.forward().cpu().numpy().tobytes() == want.tobytes()
assert ens.active_tiles()[0] > 0
""")


@pytest.mark.parametrize("graph", [True, False])
def test_ensemble_gradient_after_a_forward_that_gave_up(graph):
    fakes.run(ENSEMBLE + """
ens.set_graph(%r)
again = ens.loss_grad(target, want_h0_grad=True)
assert np.abs(again[0] - loss).max() <= 1e-13 * np.abs(loss).max()
assert np.abs(again[1] - grad).max() <= 1e-12 * np.abs(grad).max()
assert again[2].cpu().numpy().tobytes() == gh0.cpu().numpy().tobytes()
""" % graph)


def test_rollout_workspace_after_one_that_gave_up():
    fakes.run("""
import torch
from opencal_gb300 import adjoint, workloads as W
lib = adjoint._lib()
z, h = (torch.from_numpy(a).cuda() for a in W.sciddicaT_inputs(48, 56, seed=3))
hd = lib.cal_sdt_adj_create(48, 56, 31, 0)
got = []
for k in range(3):
    if k == 1:
        fake.fake_cut_at = 0
    hT = torch.empty_like(h)
    st = torch.cuda.current_stream().cuda_stream
    assert lib.cal_sdt_adj_forward(hd, z.data_ptr(), h.data_ptr(), 0.5, 0.001, hT.data_ptr(), st) == 0
    torch.cuda.synchronize()
    got.append(hT.cpu().numpy())
lib.cal_sdt_adj_destroy(hd)
assert np.isnan(got[1]).all() and got[2].tobytes() == got[0].tobytes()
""")
