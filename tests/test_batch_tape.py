"""An ensemble whose flow outgrows its tape between two evaluations: the
recorded evaluation must not outlive the tape it was recorded with.  Every
gradient against that of a fresh ensemble (whose sums of a few thousand terms
may differ in their order: 1e-12 of the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,steps", [(48, 40, 30), (96, 96, 60), (160, 150, 60)])
@pytest.mark.parametrize("mode", ["full", "segments"])
def test_flow_outgrows_the_recorded_tape(rows, cols, steps, mode):
    import opencal_gb300 as cal
    from opencal_gb300 import ensemble as E
    cal.build()
    rng = np.random.default_rng(rows)
    z = np.floor(rng.random((rows, cols)) * 2048) / 1024 + 0.125 * np.arange(rows)[:, None]
    h = np.where(rng.random((rows, cols)) < 0.3, np.floor(rng.random((rows, cols)) * 8192) / 1024, 0.0)

    def ensemble(params):
        ens = E.Ensemble([(rows, cols)] * 2, params, [z, z], [h, 0.5 * h], steps)
        ens.set_tape(mode)
        return ens

    ens = ensemble([(0.5, 6.0)] * 2)
    target = ens.pack([0.25 * h, 0.125 * h])
    needs = []
    for eps in (6.0, 4.0, 3.0, 2.0, 1.0, 0.5, 0.2, 0.05, 0.001):
        params = [(0.5, eps), (0.4, eps)]
        ens.set_params(params)
        loss, grad = ens.loss_grad(target)
        needs.append(ens.tape_info()["need_bytes"])
        fresh = ensemble(params)
        ref_loss, ref_grad = fresh.loss_grad(target)
        assert np.abs(loss - ref_loss).max() <= 1e-12 * np.abs(ref_loss).max()
        assert np.abs(grad - ref_grad).max() <= 1e-12 * np.abs(ref_grad).max()
        fresh.close()
    assert max(needs) > 2 * needs[0]
    ens.close()
