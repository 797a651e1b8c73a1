"""The work that programs built on opencal_gb300 have it do, as measured cases.

Families (``kind``), each through the entry points that a program calls:

  sdt      one SCIDDICA-T grid run from host arrays and read back
           (cal_sciddicaT_open once, then cal_sciddicaT_host_run per input),
           as its one-launch loop, with active cells, or as the reference
           program's device processes on the generic engine
  life     a model defined by a program (opencal_gb300.program): an
           elementary process compiled for the C API, loaded, run, read
  ensemble SCIDDICA-T instances of uneven sizes advanced together: scenario
           sweeps (Ensemble.forward) and calibration steps
           (Ensemble.loss_grad)
  rollout  one SCIDDICA-T rollout as a differentiable torch function,
           forward and backward
  sciara   SCIARA-fv2 eruption scenarios advanced together: hazard maps
           (SciaraBatch.run, .read) and emission-rate gradients
           (SciaraBatch.loss_grad)

Inputs follow the distributions of opencal_gb300.workloads (tilted plane with
hills and one paraboloid source; a noisy cone with vents near its summit;
Bernoulli cells), made on the GPU from the seed.  ``exact`` restates the
models in plain torch, 64 bits.
"""
import ctypes as C
import math
import random

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

import opencal_gb300 as cal
from opencal_gb300 import adjoint, ensemble
from opencal_gb300 import program as P

DEV = "cuda"


def listed():
    return [
        # a teaching-size grid: the whole call is launches and latency
        {"name": "sdt_small", "kind": "sdt", "rows": 96, "cols": 80, "steps": 100, "toroidal": True, "active": False,
         "form": "persist"},
        # the grid of the reference's shipped SCIDDICA-T data set (610 x 496, toroidal)
        {"name": "sdt_shipped", "kind": "sdt", "rows": 610, "cols": 496, "steps": 2000, "toroidal": True,
         "active": False, "form": "persist"},
        # the benchmark's grid and run length
        {"name": "sdt_large", "kind": "sdt", "rows": 2048, "cols": 2048, "steps": 4000, "toroidal": False,
         "active": False, "form": "persist"},
        # a run with the active-cells optimisation on, on a ragged grid
        {"name": "sdt_active", "kind": "sdt", "rows": 1021, "cols": 983, "steps": 1500, "toroidal": False,
         "active": True, "form": "persist"},
        # the reference program's own processes on the generic engine
        {"name": "sdt_processes", "kind": "sdt", "rows": 610, "cols": 496, "steps": 600, "toroidal": True,
         "active": False, "form": "processes"},
        # a user's own model: the grid of the Life benchmark, byte cells
        {"name": "life_program", "kind": "life", "rows": 1024, "cols": 1024, "steps": 400, "toroidal": True},
        # a first look at a calibration: few small catchments, one gradient
        {"name": "ensemble_grad_small", "kind": "ensemble", "count": 6, "lo": 96, "hi": 160, "steps": 60,
         "grad": True},
        # a calibration step of an ensemble of the sizes of the calibration benchmark
        {"name": "ensemble_grad_large", "kind": "ensemble", "count": 64, "lo": 128, "hi": 1024, "steps": 500,
         "grad": True},
        # a scenario sweep: thickness maps only
        {"name": "ensemble_forward", "kind": "ensemble", "count": 40, "lo": 128, "hi": 640, "steps": 300,
         "grad": False},
        # one catchment in an autograd program
        {"name": "rollout_grad", "kind": "rollout", "rows": 512, "cols": 480, "steps": 400, "toroidal": False},
        # hazard maps of sixteen eruptions, six hours at one minute a step
        {"name": "sciara_hazard", "kind": "sciara", "count": 16, "rows": 1024, "cols": 1000, "phases": 6,
         "grad": False},
        # emission rates from mapped thicknesses, four hours
        {"name": "sciara_grad", "kind": "sciara", "count": 16, "rows": 700, "cols": 768, "phases": 4, "grad": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sdt", "sdt", "sdt", "life", "ensemble", "ensemble", "rollout", "sciara", "sciara"])
    if kind == "sdt":
        form = rng.choice(["persist", "persist", "processes"])
        hi = 2048 if form == "persist" else 1024
        return {"kind": kind, "rows": _log(rng, 64, hi), "cols": _log(rng, 64, hi),
                "steps": _log(rng, 80, 3000 if form == "persist" else 600), "toroidal": rng.random() < 0.5,
                "active": form == "persist" and rng.random() < 0.35, "form": form}
    if kind == "life":
        return {"kind": kind, "rows": _log(rng, 64, 1500), "cols": _log(rng, 64, 1500), "steps": _log(rng, 50, 600),
                "toroidal": rng.random() < 0.6}
    if kind == "ensemble":
        lo = rng.randint(64, 160)
        return {"kind": kind, "count": _log(rng, 3, 48), "lo": lo, "hi": lo + _log(rng, 32, 700),
                "steps": _log(rng, 40, 400), "grad": rng.random() < 0.65}
    if kind == "rollout":
        return {"kind": kind, "rows": _log(rng, 96, 640), "cols": _log(rng, 96, 640), "steps": _log(rng, 40, 400),
                "toroidal": rng.random() < 0.4}
    return {"kind": kind, "count": _log(rng, 1, 16), "rows": _log(rng, 200, 900), "cols": _log(rng, 200, 900),
            "phases": rng.randint(1, 4), "grad": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------


def _quantise(x):
    return torch.floor(x * 1024.0) / 1024.0


def _hillslope(rng, rows, cols):
    """(z, h): a plane falling towards row 0 with 20 Gaussian hills, and one
    paraboloid source in the upper half, away from the edges."""
    scale = min(1.0, min(rows, cols) / 2048.0)
    margin = 300 if min(rows, cols) >= 1024 else max(4, min(rows, cols) // 4)
    ii = torch.arange(rows, dtype=torch.float64, device=DEV)
    jj = torch.arange(cols, dtype=torch.float64, device=DEV)
    z = (0.3 * ii)[:, None] + torch.zeros(cols, dtype=torch.float64, device=DEV)
    for _ in range(20):
        amp, sg = rng.uniform(10.0, 200.0), rng.uniform(20.0, 200.0) * scale
        ci, cj = rng.uniform(0.0, rows - 1.0), rng.uniform(0.0, cols - 1.0)
        gi = amp * torch.exp(-((ii - ci) ** 2) / (2.0 * sg * sg))
        gj = torch.exp(-((jj - cj) ** 2) / (2.0 * sg * sg))
        z = z + gi[:, None] * gj[None, :]
    z = _quantise(z.clamp(0.0, 2000.0))
    a, b = (max(2.0, rng.uniform(20.0, 80.0) * scale) for _ in range(2))
    depth = rng.uniform(1.0, 20.0)
    lo = max(margin + a, 0.55 * rows)
    ci = rng.uniform(lo, max(lo, rows - 1 - margin - a))
    cj = rng.uniform(margin + b, max(margin + b, cols - 1 - margin - b))
    r2 = ((ii - ci) / a)[:, None] ** 2 + ((jj - cj) / b)[None, :] ** 2
    return z, _quantise(torch.where(r2 < 1.0, depth * (1.0 - r2), torch.zeros_like(r2)))


def _physics(rng):
    """(p_r, p_eps) of one calibration instance."""
    return rng.uniform(0.3, 0.7), rng.uniform(5e-4, 5e-3)


def _instances(case, seed):
    """dims, parameters, true parameters, z and h (on the GPU) of an ensemble;
    the sizes are the case's own, whatever the seed."""
    sizes = random.Random(case["count"] * 1000003 + case["lo"] * 1009 + case["hi"])
    rng = random.Random(seed)
    dims = [(sizes.randint(case["lo"], case["hi"]), sizes.randint(case["lo"], case["hi"]))
            for _ in range(case["count"])]
    true = [_physics(rng) for _ in dims]
    start = [(r * 1.08, e * 0.92) for r, e in true]
    fields = [_hillslope(rng, r, c) for r, c in dims]
    return dims, start, true, [f[0] for f in fields], [f[1] for f in fields]


def _volcano(rng, rows, cols):
    """A cone (3000 m over 20.48 km on 10 m cells) with fractal noise of 5 m."""
    slope = 3000.0 / 20480.0
    ci, cj = (rows - 1) / 2.0, (cols - 1) / 2.0
    ii = torch.arange(rows, dtype=torch.float64, device=DEV)[:, None]
    jj = torch.arange(cols, dtype=torch.float64, device=DEV)[None, :]
    d = torch.sqrt((ii - ci) ** 2 + (jj - cj) ** 2) * 10.0
    g = torch.Generator().manual_seed(rng.randrange(1 << 31))
    noise, amp, step, total = torch.zeros(rows, cols, dtype=torch.float64, device=DEV), 1.0, 64, 0.0
    for _ in range(5):
        lattice = torch.rand(1, 1, rows // step + 2, cols // step + 2, generator=g, dtype=torch.float64) * 2.0 - 1.0
        size = ((rows // step + 2) * step, (cols // step + 2) * step)
        up = F.interpolate(lattice.to(DEV), size=size, mode="bilinear", align_corners=False)
        noise = noise + amp * up[0, 0, :rows, :cols]
        total, amp, step = total + amp, amp * 0.5, max(step // 2, 1)
    top = slope * min(rows, cols) / 2.0 * 10.0
    return _quantise(((top - slope * d).clamp(min=0.0) + 5.0 * noise / total).clamp(min=0.0))


def _eruptions(case, seed):
    """[(z on the GPU, vents [(x, y)], rates [vent][phase], 3600 s)], two
    scenarios on each volcano with vents of their own."""
    rng = random.Random(seed)
    rows, cols = case["rows"], case["cols"]
    spread, z, out = max(1.0, min(rows, cols) / 16.0), None, []
    for k in range(case["count"]):
        if k % 2 == 0:
            z = _volcano(rng, rows, cols)
        vents, count = [], 1 + (k + rows + cols) % 3
        while len(vents) < count:
            v = (int((cols - 1) / 2.0 + rng.uniform(-spread, spread)),
                 int((rows - 1) / 2.0 + rng.uniform(-spread, spread)))
            if v not in vents:
                vents.append(v)
        rates = [[rng.uniform(10.0, 50.0) for _ in range(case["phases"])] for _ in vents]
        out.append((z, vents, rates, 3600))
    return out


LIFE = (P.Program("perf_life").substates(alive="b").process("life_rule", """
    int sum = 0;
    for (int n = 1; n < ca->sizeof_X; n++)
        sum += calGetX2Db(ca, Q.alive, i, j, n);
    const CALbyte a = calGet2Db(ca, Q.alive, i, j);
    calSet2Db(ca, Q.alive, i, j, (sum == 3 || (a == 1 && sum == 2)) ? 1 : 0);
"""))

# The handle a program keeps between its runs: one at a time of each sort
# (SCIDDICA-T's substates and a program's bindings are globals of the
# library, as in the reference), opened when a run of other sizes comes.
_kept = {}


def _keep(sort, key, make, close):
    if _kept.get(sort, (None, None))[0] != key:
        if sort in _kept:
            close(_kept.pop(sort)[1])
        _kept[sort] = (key, make())
    return _kept[sort][1]


def _ptr(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double))


def _session(s):
    lib, case = s["lib"], s["case"]

    def make():
        h = lib.cal_sciddicaT_open(case["rows"], case["cols"], int(case["toroidal"]), int(case["active"]), s["p"][0],
                                   s["p"][1], _ptr(s["z"]), _ptr(s["h"]),
                                   cal.MODE_PROCESSES if case["form"] == "processes" else cal.MODE_FUSED)
        if not h:
            raise cal.CALError("cal_sciddicaT_open failed")
        return h

    key = (case["rows"], case["cols"], case["toroidal"], case["active"], case["form"])
    return _keep("session", key, make, lib.cal_sciddicaT_close)


def _life_model(case):
    def make():
        lib = LIFE.build()
        model = P.Model2D(case["rows"], case["cols"], P.CAL_MOORE_NEIGHBORHOOD_2D,
                          P.CAL_SPACE_TOROIDAL if case["toroidal"] else P.CAL_SPACE_FLAT)
        alive = model.add_substate("b")
        lib.bind(alive=alive)
        model.add_process(lib.process("life_rule"))
        return model, alive, P.Run2D(model, 1, case["steps"], graph=True)

    def close(kept):
        kept[2].close()
        kept[0].close()

    return _keep("life", (case["rows"], case["cols"], case["steps"], case["toroidal"]), make, close)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sdt":
        rng = random.Random(seed)
        p = (0.5, 0.001) if seed % 2 else _physics(rng)  # the reference's parameters, or a calibration's
        z, h = (t.cpu().pin_memory() for t in _hillslope(rng, case["rows"], case["cols"]))
        s = {"case": case, "lib": ensemble._lib(), "z": z, "h": h, "p": p, "out": torch.empty_like(h).pin_memory()}
        _session(s)
        return s
    if kind == "life":
        g = torch.Generator().manual_seed(seed)
        grid = (torch.rand(case["rows"], case["cols"], generator=g) < 0.3).numpy().astype(np.int8)
        _life_model(case)
        return {"case": case, "grid": grid}
    if kind == "ensemble":
        dims, start, true, zs, hs = _instances(case, seed)
        ens = ensemble.Ensemble(dims, true, [z.cpu().numpy() for z in zs], [h.cpu().numpy() for h in hs],
                                case["steps"])
        s = {"case": case, "ens": ens}
        if case["grad"]:  # mapped thicknesses: the run at the true parameters
            s["target"] = ens.forward()
            ens.set_params(start)
        return s
    if kind == "rollout":
        rng = random.Random(seed)
        z, h = _hillslope(rng, case["rows"], case["cols"])
        target = h * (0.2 + 0.3 * rng.random())
        p_r, p_eps = (torch.tensor(v, dtype=torch.float64, device=DEV, requires_grad=True) for v in _physics(rng))
        return {"case": case, "z": z, "h": h.clone().requires_grad_(True), "target": target, "r": p_r, "eps": p_eps}
    scenarios = _eruptions(case, seed)
    host = {}
    sb = cal.SciaraBatch([(host.setdefault(id(z), z.cpu().numpy()), v, r, et) for z, v, r, et in scenarios])
    s = {"case": case, "batch": sb}
    if case["grad"]:  # mapped thicknesses: a smooth blanket around the summit
        s["target"] = np.concatenate([t.cpu().numpy().ravel() for t in _mapped(case, seed)])
    return s


def _mapped(case, seed):
    rng = random.Random(seed + 77)
    i = torch.arange(case["rows"], dtype=torch.float64, device=DEV)[:, None] / case["rows"] - 0.5
    j = torch.arange(case["cols"], dtype=torch.float64, device=DEV)[None, :] / case["cols"] - 0.5
    return [_quantise(rng.uniform(1.0, 6.0) * torch.exp(-(i * i + j * j) * 200.0)) for _ in range(case["count"])]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sdt":
        lib, h = s["lib"], _session(s)
        lib.cal_sciddicaT_set_params(h, s["p"][0], s["p"][1])
        if lib.cal_sciddicaT_host_run(h, _ptr(s["z"]), _ptr(s["h"]), case["steps"],
                                      2 if case["form"] == "processes" else 4, _ptr(s["out"])):
            raise cal.CALError("cal_sciddicaT_host_run failed")
        return s["out"]
    if kind == "life":
        model, alive, sim = _life_model(case)
        model.load(alive, s["grid"])
        sim.run()
        return model.read(alive)
    if kind == "ensemble":
        if not case["grad"]:
            return s["ens"].forward()
        return s["ens"].loss_grad(s["target"])
    if kind == "rollout":
        leaves = (s["h"], s["r"], s["eps"])
        for t in leaves:
            t.grad = None
        hT = adjoint.rollout(s["z"], s["h"], s["r"], s["eps"], case["steps"], toroidal=case["toroidal"])
        ((hT - s["target"]) ** 2).sum().backward()
        return [hT.detach()] + [t.grad for t in leaves]
    if not case["grad"]:
        s["batch"].run()
        return s["batch"].read("slt")
    loss, grads, _ = s["batch"].loss_grad(s["target"])
    return [loss, grads]


def work(case):
    """Inputs read once, outputs written once; operations of the cells that
    can change (flowing cells estimated from the source's and the vents'
    spread), of a whole run."""
    kind, steps = case["kind"], case.get("steps", 60 * case.get("phases", 0))
    if kind in ("sdt", "rollout"):
        n = case["rows"] * case["cols"]
        wet = min(n, _film(case["rows"], case["cols"], steps))
        if kind == "sdt":
            return {"bytes": 24 * n, "flops": 40.0 * wet * steps}
        return {"bytes": 8 * 5 * n, "flops": 80.0 * wet * steps}
    if kind == "life":
        n = case["rows"] * case["cols"]
        return {"bytes": 2 * n, "flops": 10.0 * n * steps}
    if kind == "ensemble":
        mean = (case["lo"] + case["hi"]) / 2.0
        n, wet = case["count"] * mean * mean, case["count"] * min(mean * mean, _film(mean, mean, steps))
        return {"bytes": 24 * n, "flops": (80.0 if case["grad"] else 40.0) * wet * steps}
    n = case["count"] * case["rows"] * case["cols"]
    lava = case["count"] * 2 * 8.0 * steps
    return {"bytes": 16 * n, "flops": (500.0 if case["grad"] else 200.0) * lava * steps}


def _film(rows, cols, steps):
    """Flowing cells, averaged over a run: the source's disc, spreading."""
    radius = 50.0 * min(1.0, min(rows, cols) / 2048.0)
    return math.pi * radius * (radius + 0.1 * steps)


# ---- the models in plain torch, 64 bits -----------------------------------


def _flows(z, h, eps, r, idx, nbr):
    """SCIDDICA-T's minimisation at the cells idx: (kept outflows (4, k), kept mask)."""
    zh = z + h
    m = h[idx] - eps
    u = [z[idx] + eps] + [torch.where(ok, zh[at], torch.zeros_like(m)) for at, ok in nbr]
    with torch.no_grad():
        alive = torch.ones(5, len(idx), dtype=torch.bool, device=DEV)
    while True:
        avg = m
        for n in range(5):
            avg = torch.where(alive[n], avg + u[n], avg)
        count = alive.sum(0)
        avg = torch.where(count > 0, avg / count.clamp(min=1), avg)
        with torch.no_grad():
            gone = alive & (avg[None] <= torch.stack([x.detach() for x in u]))
            if not bool(gone.any()):
                break
            alive = alive & ~gone
    return torch.stack([torch.where(alive[n], (avg - u[n]) * r, torch.zeros_like(avg)) for n in range(1, 5)]), alive[1:]


def _around(idx, rows, cols, toroidal):
    """Index and presence of the north, west, east and south neighbours."""
    i, j = idx // cols, idx % cols
    out = []
    for di, dj in ((-1, 0), (0, -1), (0, 1), (1, 0)):
        a, b = i + di, j + dj
        ok = torch.ones_like(a, dtype=torch.bool) if toroidal else (a >= 0) & (a < rows) & (b >= 0) & (b < cols)
        out.append(((a % rows) * cols + b % cols, ok))
    return out


def _balance(h, f, rows, cols, toroidal):
    """h plus inflows minus outflows of every cell, in the model's order."""
    f = f.view(4, rows, cols)

    def moved(x, di, dj):
        if toroidal:
            return torch.roll(x, (di, dj), (0, 1))
        p = F.pad(x[None, None], (1, 1, 1, 1))[0, 0]
        return p[1 - di:1 - di + rows, 1 - dj:1 - dj + cols]

    inflow = [moved(f[3], 1, 0), moved(f[2], 0, 1), moved(f[1], 0, -1), moved(f[0], -1, 0)]
    x = h.view(rows, cols)
    for n in range(4):
        x = x + (inflow[n] - f[n])
    return x.reshape(-1)


def _sdt_step(z, h, eps, r, rows, cols, toroidal):
    idx = (h.detach() > eps).nonzero()[:, 0]
    f, _ = _flows(z, h, eps, r, idx, _around(idx, rows, cols, toroidal))
    full = torch.zeros(4, rows * cols, dtype=torch.float64, device=DEV).index_put(
        (torch.arange(4, device=DEV)[:, None], idx[None]), f)
    return _balance(h, full, rows, cols, toroidal)


def _sdt_start(z, h):
    return torch.where(h.detach() > 0, z - h, z).reshape(-1), h.reshape(-1)


def _sdt_run(z, h, p, steps, rows, cols, toroidal, active):
    z, h = _sdt_start(z, h)
    if not active:
        for _ in range(steps):
            h = _sdt_step(z, h, p[1], p[0], rows, cols, toroidal)
        return h.view(rows, cols)
    on, f = h > 0, torch.zeros(4, rows * cols, dtype=torch.float64, device=DEV)
    for _ in range(steps):
        idx = (on & (h > p[1])).nonzero()[:, 0]
        nbr = _around(idx, rows, cols, toroidal)
        f[:, idx], kept = _flows(z, h, p[1], p[0], idx, nbr)
        on = on.clone()
        for n, (at, ok) in enumerate(nbr):
            on[at[kept[n] & ok]] = True
        h = torch.where(on, _balance(h, f, rows, cols, toroidal), h)
        on = on & ~(h <= p[1])
        f = torch.where(on[None], torch.zeros_like(f), f)
    return h.view(rows, cols)


def _sdt_grad(z, h, r, eps, target, steps, rows, cols, toroidal):
    """Loss, h_T, dL/dh0, dL/dr, dL/deps of sum (h_T - target)^2."""
    h0 = h.detach().clone().requires_grad_(True)
    r, eps = (torch.tensor(float(v), dtype=torch.float64, device=DEV, requires_grad=True) for v in (r, eps))
    zz, x = _sdt_start(z, h0)
    for _ in range(steps):
        x = checkpoint(_sdt_step, zz, x, eps, r, rows, cols, toroidal, use_reentrant=False)
    loss = ((x.view(rows, cols) - target) ** 2).sum()
    loss.backward()
    return loss.detach(), x.detach().view(rows, cols), h0.grad, r.grad, eps.grad


MOORE = ((0, 0), (-1, 0), (0, -1), (0, 1), (1, 0), (-1, -1), (1, -1), (1, 1), (-1, 1))
OPPOSITE = (0, 4, 3, 2, 1, 7, 8, 5, 6)


def _sciara_params():
    """The 2006 configuration's values, and the power laws' coefficients."""
    clock, tsol, tvent, pr_s, pr_v, hc_s, hc_v = 60.0, 1143.0, 1360.0, 0.075, 0.90, 60.0, 0.4
    b = (math.log10(pr_v) - math.log10(pr_s)) / (tvent - tsol)
    d = (math.log10(hc_v) - math.log10(hc_s)) / (tvent - tsol)
    return {"clock": clock, "tsol": tsol, "tvent": tvent, "b": b, "a": math.log10(pr_s) - b * tsol, "d": d,
            "c": math.log10(hc_s) - d * tsol, "cool": 9.0, "rho": 2600.0, "eps": 0.90, "sigma": 5.68e-08,
            "cv": 1150.0, "w": 10.0, "ac": 100.0}


def _beside(x, k):
    """Moore neighbour k's value at every cell of (B, rows, cols); 0 outside."""
    di, dj = MOORE[k]
    p = F.pad(x, (1, 1, 1, 1))
    return p[:, 1 + di:1 + di + x.shape[1], 1 + dj:1 + dj + x.shape[2]]


def _sciara_step(z, slt, st, emit, vent, edge, q):
    """One step of every scenario; emit: thickness added at the vent cells."""
    slt = slt + emit
    st = torch.where(vent, torch.full_like(st, q["tvent"]), st)
    lava = slt.detach() > 0
    pr, hc = torch.pow(10.0, q["a"] + q["b"] * st), torch.pow(10.0, q["c"] + q["d"] * st)
    h = [slt] + [_beside(slt, k) for k in range(1, 9)]
    zk = [z] + [_beside(z, k) for k in range(1, 9)]
    for k in range(5, 9):
        zk[k] = z - (z - zk[k]) / math.sqrt(2.0)
    top = z + slt
    H = [z] + [zk[k] + h[k] for k in range(1, 9)]
    with torch.no_grad():
        kept = torch.stack([lava] + [lava & (top > H[k]) for k in range(1, 9)])
        fixed = torch.stack([x.detach() for x in H])
        drop = torch.stack([top - x for x in H])
    while True:
        avg = slt
        for k in range(9):
            avg = torch.where(kept[k], avg + H[k], avg)
        avg = avg / kept.sum(0).clamp(min=1)
        with torch.no_grad():
            gone = kept & (avg[None] <= fixed)
            if not bool(gone.any()):
                break
            kept = kept & ~gone
    with torch.no_grad():
        moves = kept & (slt[None] > hc[None] * torch.cos(torch.atan(drop / q["w"]))) & (avg[None] > fixed)
    f = [torch.where(moves[k], pr * (avg - H[k]), torch.zeros_like(avg)) for k in range(1, 9)]
    heat = inflow = outflow = torch.zeros_like(slt)
    for k in range(1, 9):
        came = _beside(f[OPPOSITE[k] - 1], k)
        heat = heat + came * _beside(st, k)
        inflow = inflow + came
        outflow = outflow + f[k - 1]
    flowing = ((inflow > 0) | (outflow > 0)).detach()
    left = slt - outflow
    mixed = (left * st + heat) / torch.where(flowing, left + inflow, torch.ones_like(left))
    st = torch.where(flowing, mixed, st)
    slt = slt + (inflow - outflow)
    hot = (slt.detach() > 0) & ~edge
    deep, warm = torch.where(hot, slt, torch.ones_like(slt)), torch.where(hot, st, torch.full_like(st, q["tvent"]))
    aus = 1.0 + 3 * warm ** 3 * q["eps"] * q["sigma"] * q["clock"] * q["cool"] / (q["rho"] * q["cv"] * deep * q["ac"])
    st = torch.where(hot, warm / torch.pow(aus, 1.0 / 3.0), st)
    solid = hot & (st.detach() <= q["tsol"])
    z = torch.where(solid, z + slt, z)
    slt = torch.where(solid | edge, torch.zeros_like(slt), slt)
    st = torch.where(solid, torch.full_like(st, q["tsol"]), st)
    return z, slt, torch.where(edge, torch.zeros_like(st), st)


class _Sciara:
    """The scenarios of a case, stepped inside a window around their lava."""

    def __init__(self, case, seed):
        self.sc = _eruptions(case, seed)
        self.q = _sciara_params()
        self.rows, self.cols = case["rows"], case["cols"]
        self.steps = 60 * case["phases"]
        self.z = torch.stack([s[0] for s in self.sc])
        self.where = [(b, y, x) for b, s in enumerate(self.sc) for x, y in s[1]]
        self.edge = torch.ones_like(self.z, dtype=torch.bool)
        self.edge[:, 1:-1, 1:-1] = False
        self.vent = torch.zeros_like(self.edge)
        for at in self.where:
            self.vent[at] = True

    def rates(self):
        return torch.tensor([r for s in self.sc for r in s[2]], dtype=torch.float64, device=DEV)

    def emission(self, rates, step, shape, i0, j0):
        at = torch.tensor(self.where, device=DEV).T
        depth = rates[:, int(step * self.q["clock"] / 3600.0)] / self.q["ac"] * self.q["clock"]
        return torch.zeros(shape, dtype=torch.float64, device=DEV).index_put((at[0], at[1] - i0, at[2] - j0), depth)

    def window(self, slt, pad):
        live = ((slt > 0) | self.vent).any(0).nonzero()
        lo, hi = live.amin(0), live.amax(0)
        return (max(0, int(lo[0]) - pad), min(self.rows, int(hi[0]) + pad + 1), max(0, int(lo[1]) - pad),
                min(self.cols, int(hi[1]) + pad + 1))

    def forward(self):
        """The final (z, slt, st) and the window of all the lava there was."""
        z, slt, st = self.z.clone(), torch.zeros_like(self.z), torch.zeros_like(self.z)
        rates, box = self.rates(), None
        with torch.no_grad():
            for first in range(0, self.steps, 10):
                i0, i1, j0, j1 = self.window(slt, 13)  # lava moves one cell a step at most
                box = (i0, i1, j0, j1) if box is None else (min(box[0], i0), max(box[1], i1), min(box[2], j0),
                                                            max(box[3], j1))
                part = [x[:, i0:i1, j0:j1].clone() for x in (z, slt, st)]
                for step in range(first, min(first + 10, self.steps)):
                    part = _sciara_step(*part, self.emission(rates, step, part[0].shape, i0, j0),
                                        self.vent[:, i0:i1, j0:j1], self.edge[:, i0:i1, j0:j1], self.q)
                for x, v in zip((z, slt, st), part):
                    x[:, i0:i1, j0:j1] = v
        return z, slt, st, box

    def grad(self, target):
        _, slt, _, (i0, i1, j0, j1) = self.forward()
        outside = ((slt - target) ** 2).sum((1, 2)) - ((slt - target)[:, i0:i1, j0:j1] ** 2).sum((1, 2))
        rates = self.rates().requires_grad_(True)
        part = [x[:, i0:i1, j0:j1].clone() for x in (self.z, torch.zeros_like(self.z), torch.zeros_like(self.z))]
        vent, edge, tgt = (x[:, i0:i1, j0:j1] for x in (self.vent, self.edge, target))
        for step in range(self.steps):
            part = checkpoint(_sciara_step, *part, self.emission(rates, step, part[0].shape, i0, j0), vent, edge,
                              self.q, use_reentrant=False)
        inside = ((part[1] - tgt) ** 2).sum((1, 2))
        inside.sum().backward()
        return (inside.detach() + outside).cpu().numpy(), rates.grad.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "sdt":
        rng = random.Random(seed)
        p = (0.5, 0.001) if seed % 2 else _physics(rng)
        z, h = _hillslope(rng, case["rows"], case["cols"])
        with torch.no_grad():
            return _sdt_run(z, h, p, case["steps"], case["rows"], case["cols"], case["toroidal"], case["active"]).cpu()
    if kind == "life":
        return None  # whole numbers
    if kind == "ensemble":
        if case["count"] * case["steps"] > (1500 if case["grad"] else 13000):
            return None  # minutes
        dims, start, true, zs, hs = _instances(case, seed)
        if case["grad"]:
            got = []
            for (rows, cols), p, t, z, h in zip(dims, start, true, zs, hs):
                with torch.no_grad():
                    target = _sdt_run(z, h, t, case["steps"], rows, cols, False, False)
                got.append(_sdt_grad(z, h, p[0], p[1], target, case["steps"], rows, cols, False))
            return (np.array([float(g[0]) for g in got]), np.array([[float(g[3]), float(g[4])] for g in got]))
        with torch.no_grad():
            parts = [_sdt_run(z, h, t, case["steps"], r, c, False, False).reshape(-1)
                     for (r, c), t, z, h in zip(dims, true, zs, hs)]
        return torch.cat([F.pad(x, (0, -len(x) % 32)) for x in parts])  # instances start at multiples of 32 cells
    if kind == "rollout":
        rng = random.Random(seed)
        rows, cols = case["rows"], case["cols"]
        z, h = _hillslope(rng, rows, cols)
        target = h * (0.2 + 0.3 * rng.random())
        p = _physics(rng)
        return list(_sdt_grad(z, h, p[0], p[1], target, case["steps"], rows, cols, case["toroidal"])[1:])
    model = _Sciara(case, seed)
    if not case["grad"]:
        return list(model.forward()[1].cpu().numpy())
    loss, rates = model.grad(torch.stack(_mapped(case, seed)))
    ends = np.cumsum([len(s[1]) for s in model.sc])
    return [loss, np.split(rates, ends[:-1])]
