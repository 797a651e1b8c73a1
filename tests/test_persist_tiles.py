"""A plain SCIDDICA-T run in cooperative launches at the sizes where the form
can go wrong: grids of one row or column, smaller than a tile or than its
ring, ragged last tiles on flat and toroidal grids, odd and even step counts
(the state ends in either buffer), flows that outgrow one tile per group in
the middle of the run (the split step takes over), and runs continued from
there.  Bit for bit as the oracle and as the per-step launches."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import opencal_gb300 as cal
    import oracle
    from opencal_gb300 import ensemble as E
    cal.build()
    oracle.build()
    return cal, oracle, E


def _inputs(rows, cols, seed):
    rng = np.random.default_rng(seed)
    z = np.floor(rng.random((rows, cols)) * 4096) / 1024 + 0.25 * np.arange(rows)[:, None]
    h = np.where(rng.random((rows, cols)) < 0.15, np.floor(rng.random((rows, cols)) * 8192) / 1024, 0.0)
    return z, h


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 40), (33, 1), (2, 3), (7, 15), (8, 16), (9, 17), (24, 31), (50, 70)])
@pytest.mark.parametrize("steps", [1, 8, 25])
def test_small_toroidal_grids(env, rows, cols, steps):
    cal, oracle, E = env
    z, h = _inputs(rows, cols, rows * 100 + cols)
    got = cal.sciddicaT(z, h, steps, toroidal=True, mode=cal.MODE_FUSED, graph=4)[1]
    per_step = cal.sciddicaT(z, h, steps, toroidal=True, mode=cal.MODE_FUSED, graph=0)[1]
    assert got.tobytes() == per_step.tobytes()
    if rows > 1 and cols > 1:
        assert got.tobytes() == oracle.sciddicaT(z, h, steps, toroidal=True, ac=False)[1].tobytes()


@pytest.mark.parametrize("rows,cols", [(1, 40), (7, 15), (9, 17), (50, 70), (129, 257)])
@pytest.mark.parametrize("steps", [1, 8, 25])
def test_flat_grids_flow_across_the_edges(env, rows, cols, steps):
    cal, _, _ = env
    z, h = _inputs(rows, cols, rows * 100 + cols)
    got = cal.sciddicaT(z, h, steps, toroidal=False, mode=cal.MODE_FUSED, graph=4)[1]
    per_step = cal.sciddicaT(z, h, steps, toroidal=False, mode=cal.MODE_FUSED, graph=0)[1]
    assert got.tobytes() == per_step.tobytes()


@pytest.mark.parametrize("rows,cols", [(17, 33), (41, 48), (49, 65), (64, 96)])
@pytest.mark.parametrize("toroidal", [0, 1])
def test_flows_that_come_to_rest(env, rows, cols, toroidal):
    """long runs: tiles of wet cells at rest leave the list and come back when
    a flow arrives, across last tiles of one row or column too"""
    cal, oracle, _ = env
    z, h = _inputs(rows, cols, rows + cols)
    z = z * 0.5
    h[rows // 4:] = 0.0
    got = cal.sciddicaT(z, h, 400, toroidal=bool(toroidal), mode=cal.MODE_FUSED, graph=4)[1]
    per_step = cal.sciddicaT(z, h, 400, toroidal=bool(toroidal), mode=cal.MODE_FUSED, graph=0)[1]
    assert got.tobytes() == per_step.tobytes()
    assert got.tobytes() == oracle.sciddicaT(z, h, 400, toroidal=bool(toroidal), ac=False)[1].tobytes()


@pytest.mark.parametrize("steps", [60, 61])
@pytest.mark.parametrize("toroidal", [0, 1])
def test_flow_outgrows_a_tile_per_group(env, steps, toroidal):
    """384 x 400 cells are 1200 tiles of 16 x 8, twice the groups; the source
    covers about 400 of them and spreads"""
    cal, oracle, E = env
    rows, cols = 384, 400
    i, j = np.arange(rows)[:, None], np.arange(cols)[None, :]
    z = np.floor((0.3 * i + 0.05 * j) * 1024) / 1024
    r2 = ((i - 192) / 110.0) ** 2 + ((j - 200) / 110.0) ** 2
    h = np.floor(np.where(r2 < 1.0, 9.0 * (1.0 - r2), 0.0) * 1024) / 1024
    ref = oracle.sciddicaT(z, h, steps, toroidal=bool(toroidal), ac=False)[1]
    lib = E._lib()
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    sess = lib.cal_sciddicaT_open(rows, cols, toroidal, 0, 0.5, 0.001, ptr(z), ptr(h), cal.MODE_FUSED)
    assert sess
    try:
        out = np.empty_like(h)
        for parts in ((steps,), (steps - 20, 20), (15, steps - 15)):
            lib.cal_sciddicaT_reset(sess)
            for n in parts:
                assert lib.cal_sciddicaT_steps(sess, n, 4) == 0
            assert lib.cal_sciddicaT_persist_failed(sess) == 0
            assert lib.cal_sciddicaT_read(sess, ptr(out)) == 0
            assert out.tobytes() == ref.tobytes()
    finally:
        lib.cal_sciddicaT_close(sess)
