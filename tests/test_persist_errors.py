"""What a persistent SCIDDICA-T run answers when device memory, a cooperative
launch or a grid barrier fails it: the state of the requested step, or an
error."""
import fakes
import pytest

pytestmark = pytest.mark.gpu

SESSION = """
import opencal_gb300 as cal, oracle
from opencal_gb300 import ensemble as E, workloads as W
oracle.build()
lib = E._lib()
ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
rows, cols, steps = {rows}, {cols}, 40
z, h = W.sciddicaT_inputs(rows, cols, seed=5)
ref = oracle.sciddicaT(z, h, steps, toroidal=False, ac={ac})[1]
def session():
    s = lib.cal_sciddicaT_open(rows, cols, 0, {ac}, 0.5, 0.001, ptr(z), ptr(h), cal.MODE_FUSED)
    assert s
    return s
def host_run(s):
    out = np.full_like(h, -1.0)
    rc = lib.cal_sciddicaT_host_run(s, ptr(z), ptr(h), steps, 4, ptr(out))
    return rc, out.tobytes() == ref.tobytes()
"""


# fewer tiles than the GPU has groups, and more
@pytest.mark.parametrize("rows,cols", [(96, 80), (400, 400)])
@pytest.mark.parametrize("ac", [0, 1])
def test_refused_launch_is_an_error(rows, cols, ac):
    out = fakes.run(SESSION.format(rows=rows, cols=cols, ac=ac) + """
s = session()
assert host_run(s) == (0, True)
for at in range(3):
    fake.fake_launches = 0
    fake.fake_launch_at = at
    rc, same = host_run(s)
    refused = fake.fake_launch_at == -1 and fake.fake_launches > at
    fake.fake_launch_at = -1
    assert (rc != 0) if refused else (rc == 0 and same), (at, rc, same)
    print("refused", refused)
    cal.core().calClearError()
    assert host_run(s) == (0, True)  # and the session is usable
    lib.cal_sciddicaT_close(s)
    fake.fake_launch_at = -2
    try:
        cal.sciddicaT(z, h, steps, toroidal=False, ac=bool({ac}), mode=cal.MODE_FUSED, graph=4)
        raise SystemExit("no error")
    except cal.CALError:
        pass
    fake.fake_launch_at = -1
    cal.core().calClearError()
    s = session()
lib.cal_sciddicaT_close(s)
""".replace("{ac}", str(ac)))
    assert "refused True" in out


@pytest.mark.parametrize("rows,cols", [(96, 80), (400, 400)])
def test_refused_memory_is_the_result_or_an_error(rows, cols):
    fakes.run(SESSION.format(rows=rows, cols=cols, ac=0) + """
for at in range(20):
    s = session()
    fake.fake_malloc_at = at
    rc, same = host_run(s)
    left = fake.fake_malloc_at
    fake.fake_malloc_at = -1
    cal.core().calClearError()
    if left < 0 and at < 7:  # the tile form's arrays: the run goes without them
        assert rc == 0 and same, (at, rc, same)
    assert rc != 0 or same, (at, rc, same)
    assert host_run(s) == (0, True)
    lib.cal_sciddicaT_close(s)
""")


@pytest.mark.parametrize("ac", [0, 1])
def test_barrier_that_gave_up_is_an_error(ac):
    fakes.run(SESSION.format(rows=96, cols=80, ac=ac) + """
s = session()
assert host_run(s) == (0, True)
fake.fake_read4 = 1
assert host_run(s)[0] != 0
fake.fake_read4 = 0
cal.core().calClearError()
assert host_run(s) == (0, True)
lib.cal_sciddicaT_close(s)
""")
