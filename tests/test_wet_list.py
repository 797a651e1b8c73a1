"""The wet-cell list of the rollouts and ensembles at the sizes where it can
go wrong: ragged and one-cell-thin last tiles, flat and toroidal grids, long
runs in which cells come to rest and are reached by a flow again.  Forward bit
for bit as the oracle; gradients against autograd over a plain fp64 step (the
sums of a few thousand terms of one sign differ in their order: 1e-10)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch

    import opencal_gb300 as cal
    import oracle
    from opencal_gb300 import ensemble as E
    cal.build()
    oracle.build()
    return torch, cal, oracle, E


def _inputs(rows, cols):
    rng = np.random.default_rng(rows * 100 + cols)
    z = np.floor(rng.random((rows, cols)) * 2048) / 1024 + 0.125 * np.arange(rows)[:, None]
    h = np.where(rng.random((rows, cols)) < 0.3, np.floor(rng.random((rows, cols)) * 8192) / 1024, 0.0)
    h[max(1, rows // 3):] = 0.0
    return z, h


def _beside(torch, x, q, toroidal):
    """von Neumann neighbour q's value at every cell, 0 outside a flat grid"""
    di, dj = ((-1, 0), (0, -1), (0, 1), (1, 0))[q]
    if toroidal:
        return torch.roll(x, (-di, -dj), (0, 1))
    p = torch.nn.functional.pad(x, (1, 1, 1, 1))
    return p[1 + di:1 + di + x.shape[0], 1 + dj:1 + dj + x.shape[1]]


def _step(torch, z, h, r, eps, toroidal):
    wet = ~(h.detach() <= eps.detach())
    m = h - eps
    u = [z + eps] + [_beside(torch, z + h, q, toroidal) for q in range(4)]
    elim = [torch.zeros_like(wet) for _ in range(5)]
    again = True
    while again:
        again = False
        average, count = m, torch.zeros_like(h)
        for n in range(5):
            average = average + torch.where(elim[n], 0.0, u[n])
            count = count + (~elim[n])
        average = torch.where(count > 0, average / count.clamp(min=1), average)
        for n in range(5):
            out = ~elim[n] & (average.detach() <= u[n].detach())
            again = again or bool((out & wet).any())
            elim[n] = elim[n] | out
    f = [torch.where(wet & ~elim[n + 1], (average - u[n + 1]) * r, 0.0) for n in range(4)]
    for q in range(4):
        h = h + (_beside(torch, f[3 - q], q, toroidal) - f[q])
    return h


def _reference(torch, z, h, r, eps, target, steps, toroidal):
    h0 = torch.from_numpy(h).requires_grad_(True)
    rt, et = (torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in (r, eps))
    x, zz = h0, torch.where(h0.detach() > 0, torch.from_numpy(z) - h0, torch.from_numpy(z))
    for _ in range(steps):
        x = _step(torch, zz, x, rt, et, toroidal)
    loss = ((x - torch.from_numpy(target)) ** 2).sum()
    loss.backward()
    return x.detach().numpy(), h0.grad.numpy(), float(rt.grad), float(et.grad)


def _close(a, b, rel):
    return np.abs(np.asarray(a) - np.asarray(b)).max() <= rel * max(np.abs(np.asarray(b)).max(), 1e-300)


SIZES = [(2, 3), (9, 17), (17, 33), (40, 31), (49, 65)]


@pytest.mark.parametrize("toroidal", [False, True])
@pytest.mark.parametrize("rows,cols", SIZES)
def test_rollout_comes_to_rest_as_the_oracle(env, rows, cols, toroidal):
    torch, cal, oracle, _ = env
    z, h = _inputs(rows, cols)
    zt, ht = torch.from_numpy(z).cuda(), torch.from_numpy(h).cuda()
    for steps in (1, 7, 300):
        ref = oracle.sciddicaT(z, h, steps, toroidal=toroidal, ac=False)[1]
        assert cal.adjoint.rollout(zt, ht, 0.5, 0.001, steps, toroidal).cpu().numpy().tobytes() == ref.tobytes()


@pytest.mark.parametrize("toroidal", [False, True])
@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("r", [0.5, 0.0])
def test_gradients_of_cells_at_rest(env, rows, cols, toroidal, r):
    """r = 0: nothing ever moves, and every step has its part of dL/dr"""
    torch, cal, _, _ = env
    steps, eps = 60, 0.001
    z, h = _inputs(rows, cols)
    target = h * 0.25
    hT, gh, gr, ge = _reference(torch, z, h, r, eps, target, steps, toroidal)
    h0 = torch.from_numpy(h).cuda().requires_grad_(True)
    pr, pe = (torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in (r, eps))
    x = cal.adjoint.rollout(torch.from_numpy(z).cuda(), h0, pr, pe, steps, toroidal)
    ((x - torch.from_numpy(target).cuda()) ** 2).sum().backward()
    assert _close(x.detach().cpu().numpy(), hT, 1e-12)
    assert _close(h0.grad.cpu().numpy(), gh, 1e-10)
    assert abs(float(pr.grad) - gr) <= 1e-10 * max(abs(gr), np.abs(gh).max())
    assert abs(float(pe.grad) - ge) <= 1e-10 * max(abs(ge), np.abs(gh).max())


def test_backward_after_a_forward_without_tape(env):
    torch, cal, _, _ = env
    rows, cols, steps = 40, 31, 50
    z, h = (torch.from_numpy(a).cuda() for a in _inputs(rows, cols))
    lib = cal.adjoint._lib()
    got = []
    for tape in (1, 0):
        hd = lib.cal_sdt_adj_create(rows, cols, steps, 0)
        assert hd
        try:
            lib.cal_sdt_adj_set_tape(hd, tape)
            hT, g = torch.empty_like(h), torch.empty_like(h)
            st = torch.cuda.current_stream().cuda_stream
            assert lib.cal_sdt_adj_forward(hd, z.data_ptr(), h.data_ptr(), 0.5, 0.001, hT.data_ptr(), st) == 0
            gr, ge = C.c_double(), C.c_double()
            assert lib.cal_sdt_adj_backward(hd, hT.data_ptr(), g.data_ptr(), C.byref(gr), C.byref(ge), st) == 0
            torch.cuda.synchronize()
            got.append((hT.cpu().numpy(), g.cpu().numpy(), gr.value, ge.value))
        finally:
            lib.cal_sdt_adj_destroy(hd)
    assert got[0][0].tobytes() == got[1][0].tobytes() and got[0][1].tobytes() == got[1][1].tobytes()
    assert _close(got[0][2], got[1][2], 1e-12) and _close(got[0][3], got[1][3], 1e-12)


@pytest.mark.parametrize("mode", ["full", "segments"])
def test_ensemble_comes_to_rest(env, mode):
    torch, _, oracle, E = env
    steps, eps = 120, 0.001
    zs, hs = zip(*(_inputs(r, c) for r, c in SIZES))
    params = [(0.5, eps)] * len(SIZES)
    ens = E.Ensemble(list(SIZES), params, list(zs), list(hs), steps)
    for g, z, h in zip(ens.unpack(ens.forward()), zs, hs):
        assert g.tobytes() == oracle.sciddicaT(z, h, steps, toroidal=False, ac=False)[1].tobytes()
    ens.set_tape(mode)
    out = ens.loss_grad(ens.pack([0.25 * h for h in hs]))
    grad = out[1].cpu().numpy() if torch.is_tensor(out[1]) else np.asarray(out[1])
    for b, (z, h) in enumerate(zip(zs, hs)):
        _, gh, gr, ge = _reference(torch, z, h, 0.5, eps, 0.25 * h, steps, False)
        assert abs(grad.reshape(len(SIZES), 2)[b, 0] - gr) <= 1e-10 * max(abs(gr), np.abs(gh).max())
        assert abs(grad.reshape(len(SIZES), 2)[b, 1] - ge) <= 1e-10 * max(abs(ge), np.abs(gh).max())
