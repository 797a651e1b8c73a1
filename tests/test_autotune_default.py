"""The tile shape tuner times the shape an ensemble starts with, and leaves it
with the fastest of those it timed."""
import pytest

from opencal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("probe", [0, 1, 30])
def test_default_shape_is_a_candidate(graph, probe):
    import opencal_gb300 as cal
    import oracle
    from opencal_gb300 import ensemble as E
    cal.build()
    oracle.build()
    dims = [(48, 56), (33, 140)]
    zh = [W.sciddicaT_inputs(r, c, seed=3) for r, c in dims]
    ens = E.Ensemble(dims, [(0.5, 0.001)] * 2, [z for z, _ in zh], [h for _, h in zh], 31)
    default = E.SHAPES[ens._lib.cal_sdt_batch_shape(ens.handle)]
    ens.set_graph(graph)
    name, ms = ens.autotune(probe)
    assert default in ms and ms[name] == min(ms.values()) > 0
    assert E.SHAPES[ens._lib.cal_sdt_batch_shape(ens.handle)] == name
    for got, (z, h) in zip(ens.unpack(ens.forward()), zh):
        assert got.tobytes() == oracle.sciddicaT(z, h, 31, toroidal=False, ac=False)[1].tobytes()
