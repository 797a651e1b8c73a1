"""The process kernels' cell views and the tile-wise update at the sizes where
they can go wrong: grids smaller than a tile or than the neighbourhood's
reach, one cell more or less than a tile, ragged last tiles, more tiles than
one pass of the update lists.  A process that reads its own neighbours (the
offset form inside the grid, wrapped or absent at the edges) and another
cell's neighbours (always the general form), on bytes (rows of a tile on one
block) and reals (rows spread over the blocks), against numpy: whole numbers
and exact sums, equal bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BODY = """
    int sum = 0;
    CALreal x = 0.0;
    const int a = (i + 1) % ca->rows, b = (j + 3) % ca->columns;
    for (int n = 1; n < ca->sizeof_X; n++) {
        sum += (n + 1) * calGetX2Db(ca, Q.s, i, j, n) + calGetX2Db(ca, Q.s, a, b, n);
        x += calGetX2Dr(ca, Q.v, i, j, n) + 2.0 * calGetX2Dr(ca, Q.v, a, b, n);
    }
    const int next = (sum + calGet2Db(ca, Q.s, i, j)) % 5;
    if (next != calGet2Db(ca, Q.s, i, j))
        calSet2Db(ca, Q.s, i, j, next);
    if (P.real && x != 0.0)
        calSet2Dr(ca, Q.v, i, j, x / 1024.0);
"""
BYTES = """
    int sum = 0;
    const int a = (i + 1) % ca->rows, b = (j + 3) % ca->columns;
    for (int n = 1; n < ca->sizeof_X; n++)
        sum += (n + 1) * calGetX2Db(ca, Q.s, i, j, n) + calGetX2Db(ca, Q.s, a, b, n);
    const int next = (sum + calGet2Db(ca, Q.s, i, j)) % 5;
    if (next != calGet2Db(ca, Q.s, i, j))
        calSet2Db(ca, Q.s, i, j, next);
"""
VN = [(-1, 0), (0, -1), (0, 1), (1, 0)]
MOORE = VN + [(-1, -1), (1, -1), (1, 1), (-1, 1)]


@pytest.fixture(scope="module")
def P():
    import opencal_gb300 as cal
    from opencal_gb300 import program
    cal.build()
    return program


def _beside(x, d, toroidal):
    if toroidal:
        return np.roll(x, (-d[0], -d[1]), (0, 1))
    p = np.pad(x, 1)
    return p[1 + d[0]:1 + d[0] + x.shape[0], 1 + d[1]:1 + d[1] + x.shape[1]]


def _reference(s, v, nbrs, toroidal, steps):
    for _ in range(steps):
        total = np.zeros(s.shape, np.int64)
        x = np.zeros(s.shape)
        for n, d in enumerate(nbrs):
            ns, nv = _beside(s, d, toroidal), _beside(v, d, toroidal)
            total += (n + 2) * ns.astype(np.int64) + np.roll(ns, (-1, -3), (0, 1))
            x = x + (nv + 2.0 * np.roll(nv, (-1, -3), (0, 1)))
        s = ((total + s) % 5).astype(np.int8)
        v = np.where(x != 0.0, x / 1024.0, v)
    return s, v


SIZES = [(1, 1), (1, 70), (3, 2), (7, 31), (8, 32), (9, 33), (16, 64), (65, 257), (130, 1030), (700, 900)]


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("toroidal", [0, 1])
@pytest.mark.parametrize("moore", [0, 1])
@pytest.mark.parametrize("real", [0, 1])
def test_neighbour_reads_and_tile_updates(P, rows, cols, toroidal, moore, real):
    if real:
        prog = P.Program("tiles_r").substates(s="b", v="r").parameters(real="i").process("rule", BODY)
    else:
        prog = P.Program("tiles_b").substates(s="b").process("rule", BYTES)
    lib = prog.build()
    rng = np.random.default_rng(rows * 7 + cols)
    s0 = rng.integers(0, 3, (rows, cols)).astype(np.int8) * (rng.random((rows, cols)) < 0.2)
    v0 = rng.integers(0, 9, (rows, cols)) * 0.25
    steps = 3  # sums of a few 2^-32 multiples below 2^20: every order gives the same double
    with P.Model2D(rows, cols, P.CAL_MOORE_NEIGHBORHOOD_2D if moore else P.CAL_VON_NEUMANN_NEIGHBORHOOD_2D,
                   P.CAL_SPACE_TOROIDAL if toroidal else P.CAL_SPACE_FLAT) as model:
        s = model.add_substate("b")
        if real:
            v = model.add_substate("r")
            lib.bind(s=s, v=v)
            lib.set(real=1)
        else:
            lib.bind(s=s)
        model.add_process(lib.process("rule"))
        model.load(s, s0)
        if real:
            model.load(v, v0)
        run = P.Run2D(model, 1, steps, graph=True)
        run.run()
        got = model.read(s), (model.read(v) if real else None)
        run.close()
    want = _reference(s0, v0, MOORE if moore else VN, toroidal, steps)
    assert np.array_equal(got[0], want[0])
    if real:
        assert got[1].tobytes() == want[1].tobytes()
