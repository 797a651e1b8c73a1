"""Persistent SCIDDICA-T runs a few steps a call on grids with more tiles than
the GPU has groups: the split step's lists go from call to call."""
import fakes
import pytest

pytestmark = pytest.mark.gpu

SESSION = """
import opencal_gb300 as cal, oracle
from opencal_gb300 import ensemble as E, workloads as W
oracle.build()
lib = E._lib()
ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
z, h = W.sciddicaT_inputs(400, 392, seed=5)
s = lib.cal_sciddicaT_open(400, 392, {tor}, 0, 0.5, 0.001, ptr(z), ptr(h), cal.MODE_FUSED)
assert s
out = np.empty_like(h)
def steps(n, loop=4):
    fake.fake_launches = 0
    assert lib.cal_sciddicaT_steps(s, n, loop) == 0 and lib.cal_sciddicaT_persist_failed(s) == 0
    assert lib.cal_sciddicaT_read(s, ptr(out)) == 0
    return fake.fake_launches
"""


@pytest.mark.parametrize("tor", [0, 1])
def test_short_calls_go_on_with_the_lists(tor):
    fakes.run(SESSION.format(tor=tor) + """
done = 0
for n, loop in ((1, 4), (7, 4), (43, 4), (44, 4), (2, 4), (3, 0), (60, 4), (5, 1), (1, 4), (100, 4), (4, 4)):
    launches = steps(n, loop)
    done += n
    if loop == 4:
        assert launches == (1 if n < 43 else 2), (n, launches)
    ref = oracle.sciddicaT(z, h, done, toroidal=bool(%d), ac=False)[1]
    assert out.tobytes() == ref.tobytes(), done
lib.cal_sciddicaT_close(s)
""" % tor)


@pytest.mark.parametrize("loop", [0, 4])
def test_lists_are_made_again_for_another_epsilon(loop):
    """from epsilon 0.25 to 0.001 and back, against every cell's own step"""
    fakes.run(SESSION.format(tor=0) + """
def plain(z, h, eps, n):
    zp = np.pad(z, 1)
    for _ in range(n):
        hp = np.pad(h, 1)
        u = [z + eps] + [(zp + hp)[1 + a:401 + a, 1 + b:393 + b] for a, b in ((-1, 0), (0, -1), (0, 1), (1, 0))]
        out = np.zeros((5,) + h.shape, bool)
        again = True
        while again:
            again = False
            average, count = h - eps, np.zeros(h.shape)
            for k in range(5):
                average = np.where(out[k], average, average + u[k])
                count += ~out[k]
            average = np.where(count > 0, average / np.maximum(count, 1), average)
            for k in range(5):
                drop = ~out[k] & (average <= u[k])
                again = again or (drop & (h > eps)).any()
                out[k] |= drop
        f = [np.pad(np.where((h > eps) & ~out[k + 1], (average - u[k + 1]) * 0.5, 0.0), 1) for k in range(4)]
        new = h.copy()
        for k, (a, b) in enumerate(((-1, 0), (0, -1), (0, 1), (1, 0))):
            new += f[3 - k][1 + a:401 + a, 1 + b:393 + b] - f[k][1:401, 1:393]
        h = new
    return h
z1, x = np.where(h > 0, z - h, z), h + 0.0
for eps in (0.001, 0.25, 0.001):
    lib.cal_sciddicaT_set_params(s, 0.5, eps)
    steps(6, %d)
    x = plain(z1, x, eps, 6)
    assert out.tobytes() == x.tobytes(), eps
lib.cal_sciddicaT_close(s)
""" % loop)
