"""An ensemble whose new tile shape did not fit in memory answers errors until
another shape fits."""
import fakes
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0, 1, 2])
def test_shape_that_did_not_fit(at):
    fakes.run("""
import opencal_gb300 as cal
from opencal_gb300 import ensemble as E, workloads as W
dims = [(48, 56), (33, 40)]
zh = [W.sciddicaT_inputs(r, c, seed=3) for r, c in dims]
ens = E.Ensemble(dims, [(0.5, 0.001)] * 2, [z for z, _ in zh], [h for _, h in zh], 31)
want = ens.forward().cpu().numpy()
target = ens.pack([0.5 * h for _, h in zh])
loss, grad = ens.loss_grad(target)
fake.fake_malloc_at = %d
def refused(f):
    try:
        f()
    except cal.CALError:
        return True
assert refused(lambda: ens.set_shape("16x8"))
assert refused(ens.forward) and refused(lambda: ens.loss_grad(target))
ens.set_shape("32x16")
assert ens.forward().cpu().numpy().tobytes() == want.tobytes()
again = ens.loss_grad(target)
assert np.abs(again[1] - grad).max() <= 1e-12 * np.abs(grad).max()
""" % at)
