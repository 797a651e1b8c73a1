"""SciaraBatch.loss_grad where the run's tape does not fit: taped and swept in
stretches of steps, with the gradients of the whole tape (sums by FP64
atomics: equal up to their order) and the run's final state."""
import ctypes as C

import numpy as np
import pytest

from opencal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch():
    import opencal_gb300 as cal
    cal.build()
    scs = []
    for k, (r, c) in enumerate([(48, 64), (60, 52)]):
        z, vents, rates = W.sciara_inputs(r, c, seed=40 + k, phases=3)
        scs.append((z, vents, rates, 1200))
    sb = cal.SciaraBatch(scs)
    sb._m.cal_sciara_batch_set_tape_limit.argtypes = [C.c_void_p, C.c_longlong]
    target = np.zeros(sb.cells)
    steps, _ = sb.run()
    return cal, sb, target, steps, [x.tobytes() for x in sb.read("slt")], sb.loss_grad(target)


def _limit(sb, entries):
    assert sb._m.cal_sciara_batch_set_tape_limit(sb._h, entries) == 0


@pytest.mark.parametrize("entries", [40000, 20000, 4000, 700])
def test_stretches(batch, entries):
    cal, sb, target, steps, slt, whole = batch
    sb.run()
    lava = sb.lava_cells()  # the last step's entries are these cells and more
    _limit(sb, entries)
    try:
        if entries < lava:
            with pytest.raises(cal.CALError):
                sb.loss_grad(target)
            return
        got = sb.loss_grad(target)
        np.testing.assert_allclose(got[0], whole[0], rtol=1e-12)
        for a, b in zip(got[1], whole[1]):
            np.testing.assert_allclose(a, b, rtol=1e-10, atol=1e-14)
        assert [x.tobytes() for x in sb.read("slt")] == slt
    finally:
        _limit(sb, 0)


def test_a_step_that_does_not_fit_is_an_error(batch):
    cal, sb, target, steps, slt, whole = batch
    _limit(sb, 1)
    with pytest.raises(cal.CALError):
        sb.loss_grad(target)
    _limit(sb, 0)
    np.testing.assert_allclose(sb.loss_grad(target)[0], whole[0], rtol=1e-12)
    assert sb._m.cal_sciara_batch_set_tape_limit(sb._h, -1) != 0
