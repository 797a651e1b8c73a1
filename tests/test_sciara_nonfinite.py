"""Lava at a temperature that is not finite: the split step spreads it as the
device-process program does, whose sums take 0 x t from every neighbour."""
import ctypes as C

import numpy as np
import pytest

from opencal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, -np.inf, np.inf])
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_spreads_as_the_device_processes(bad, steps):
    import opencal_gb300 as cal
    cal.build()
    rows, cols, et = 40, 48, 600
    z, vents, rates = W.sciara_inputs(rows, cols, seed=3)
    rng = np.random.default_rng(1)
    slt, st = np.zeros_like(z), np.zeros_like(z)
    slt[8:30, 8:40] = 1.0 + 4.0 * rng.random((22, 32))
    st[8:30, 8:40] = 1250.0 + 100.0 * rng.random((22, 32))
    for i, j in ((12, 12), (12, 20), (20, 15), (25, 33), (25, 34), (8, 8)):
        st[i, j] = bad
    ref = cal.sciara(z, vents, rates, et, steps, ac=False, slt0=slt, st0=st)
    sb = cal.SciaraBatch([(z, vents, rates, et)])  # its shapes and prototypes; the state below comes with st0
    h, sb._h = sb._h, None
    m = sb._m
    m.cal_sciara_batch_destroy(h)
    dims = np.array([rows, cols], np.int32)
    par = np.ascontiguousarray(W.SCIARA_PARAMS, dtype=np.float64)
    vi = np.zeros(len(vents), np.int32)
    vxy = np.ascontiguousarray(np.asarray(vents, np.int32).reshape(-1))
    rr = np.ascontiguousarray(np.asarray(rates, np.float64).reshape(-1))
    sb._h = m.cal_sciara_batch_create(1, dims.ctypes.data, z.ctypes.data, slt.ctypes.data, st.ctypes.data,
                                      par.ctypes.data, len(vents), vi.ctypes.data, vxy.ctypes.data, et,
                                      len(rates[0]), rr.ctypes.data, 0.0)
    assert sb._h
    sb.run(steps)
    (got,) = sb.read()
    for k in ("z", "slt", "st", "msl"):
        assert np.array_equal(got[k], ref[k], equal_nan=True), (k, int((got[k] != ref[k]).sum()))
    if not np.isfinite(bad):
        assert np.isnan(ref["st"]).sum() > 6 or bad == -np.inf
