"""Performance cases of the propagator, the Parareal drivers and the adjoint.

Each case goes through the public Python interface as a user's program does:
the handle and the fields are made in prepare(), run() is one call (or the few
calls that belong together) and its results.  The sizes are those of the
repository's drivers, tests and benchmark (16^3 to 256^3, cubes and ragged
boxes), with step counts cut so that a pass stays below a quarter second.

A handle is used as constructed unless the case has "tune": then the program
sets the launch shapes that an earlier sp_autotune on the same grid chose, as
the benchmark does for the instances of a batch.
"""
import math
import random

import torch

import stencilparareal_b200 as sp
from stencilparareal_b200.adjoint import misfit_gradient, rk4_propagate
from stencilparareal_b200.parareal import PararealBatch

DEVICE = 0
RK4_REACH = 2.78  # RK4's stability limit on both axes, roughly
BATCH_SIZES = (32, 48, 64)


def listed():
    base = dict(prec="f64", nufreq=0.0, nu=0.01, cx=1.0, cy=1.0, cz=1.0, upwind=True, tune="")
    paper = dict(base, nu=0.1)
    return [
        # one DoRK4Timestep on a small field: the latency of the smallest call
        dict(base, name="step_24", kind="rk4", ni=24, nj=24, nk=24, steps=1, errors=False),
        # the serial fine run of a small field, 32^3 x 1000 steps, in one call
        dict(base, name="rk4_32", kind="rk4", ni=32, nj=32, nk=32, steps=1000, errors=False),
        # a row of the reference's stability sweep: nu(t) varies, then the errors against a reference field
        dict(paper, name="rk4_100_nufreq", kind="rk4", ni=100, nj=100, nk=100, steps=100, nufreq=100.0, errors=True),
        # the fine-propagator benchmark field on the shapes its autotuner picks
        dict(base, name="rk4_256", kind="rk4", ni=256, nj=256, nk=256, steps=40, nu=1e-3, cy=0.5, cz=0.25,
             tune="pairs", errors=False),
        # the coarse propagator's precision on a ragged box
        dict(base, name="rk4_f32_ragged", kind="rk4", ni=95, nj=97, nk=93, steps=100, prec="f32", cy=-0.5,
             errors=False),
        # the reference's coarse propagator (upwind Euler) as a serial run
        dict(paper, name="euler_128", kind="euler", ni=128, nj=128, nk=128, steps=64, errors=False),
        # host arrays in and out: what a caller without device memory pays end to end
        dict(base, name="host_128", kind="host", ni=128, nj=128, nk=128, steps=200),
        # the reference's convergence experiment in small: Euler coarse, nu(t), fixed kmax
        dict(paper, name="parareal_euler_64", kind="parareal", n=64, slices=16, fine=64, coarse=8, kmax=3,
             nufreq=100.0, g="euler", gprec="f64"),
        # Parareal with an FP32 RK4 coarse propagator at the benchmark's grid and slice count
        dict(base, name="parareal_rk4_128", kind="parareal", n=128, slices=32, fine=40, coarse=7, kmax=2, g="rk4",
             gprec="f32", tune="pairs"),
        # many small independent solves of uneven grids and slice counts
        dict(base, name="batch_6", kind="batch", instances=6, fine=40, coarse=5, kmax=2, mix=1),
        # the gradient of a terminal misfit, 128^3 as in the benchmark
        dict(base, name="gradient_128", kind="gradient", ni=128, nj=128, nk=128, steps=40, every=10),
        # forward and backward through the autograd function, as an optimiser's step
        dict(base, name="autograd_48", kind="autograd", ni=48, nj=48, nk=48, steps=50, every=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rk4", "rk4", "rk4", "euler", "host", "parareal", "parareal", "batch", "gradient", "autograd"])
    c = dict(kind=kind, prec="f64", nufreq=rng.choice([0.0, 0.0, 100.0]), nu=10 ** rng.uniform(-4, -1),
             cx=rng.uniform(-1, 1), cy=rng.uniform(-1, 1), cz=rng.uniform(-1, 1), upwind=rng.random() < 0.8, tune="")

    def box(lo, hi):
        n = _log_int(rng, lo, hi)
        if rng.random() < 0.5:
            return dict(ni=n, nj=n, nk=n)
        return {k: max(8, int(round(n * rng.uniform(0.6, 1.25)))) for k in ("ni", "nj", "nk")}

    def steps(cells, budget, most):
        return max(1, min(_log_int(rng, 1, most), budget // cells))

    if kind in ("rk4", "euler"):
        c.update(box(16, 200), prec=rng.choice(["f64", "f64", "f32"]), errors=False)
        c["steps"] = steps(c["ni"] * c["nj"] * c["nk"], 400_000_000, 1000)
        if c["prec"] == "f64":
            c["errors"] = rng.random() < 0.3
            if kind == "rk4" and rng.random() < 0.3:
                c["tune"] = "pairs"
    elif kind == "host":
        c.update(box(16, 144))
        c["steps"] = steps(c["ni"] * c["nj"] * c["nk"], 200_000_000, 400)
    elif kind == "parareal":
        n, slices = _log_int(rng, 24, 112), rng.randint(4, 24)
        fine = max(8, min(_log_int(rng, 8, 96), 400_000_000 // (n ** 3 * slices)))
        c.update(n=n, slices=slices, fine=fine, coarse=rng.randint(1, 8), kmax=rng.randint(1, min(4, slices)))
        c["g"], c["gprec"] = rng.choice([("euler", "f64"), ("euler", "f32"), ("rk4", "f32"), ("rk4", "f64")])
    elif kind == "batch":
        c.update(instances=rng.randint(2, 8), fine=rng.randint(8, 40), coarse=rng.randint(2, 6),
                 kmax=rng.randint(1, 2), mix=rng.randint(2, 1 << 20), nufreq=0.0)
    else:
        c.update(box(16, 112 if kind == "gradient" else 64))
        c["steps"] = steps(c["ni"] * c["nj"] * c["nk"], 80_000_000, 100)
        c["every"] = rng.choice([0, 0, 5, 10])
    return c


# ---------------------------------------------------------------------------
# Inputs.

def _rate(c, dx):
    """The largest eigenvalue of the fourth-order right-hand side, roughly."""
    return (abs(c["cx"]) + abs(c["cy"]) + abs(c["cz"])) * 1.5 / dx + 1.5 * c["nu"] * 16.0 / (dx * dx)


def _rate2(c, dx):
    return (abs(c["cx"]) + abs(c["cy"]) + abs(c["cz"])) * 2.0 / dx + 1.5 * c["nu"] * 12.0 / (dx * dx)


def _dt(c, ni, coarse=False):
    """A step inside the stability limit of the scheme that takes it."""
    dx = 1.0 / ni
    euler = c["kind"] == "euler" or (coarse and c.get("g") == "euler")
    return 0.25 * (1.0 / _rate2(c, dx) if euler else RK4_REACH / _rate(c, dx))


def _field(seed, salt, nk, nj, ni):
    """Four random Fourier modes (wavenumbers 1-4) plus noise of amplitude 1e-3."""
    g = torch.Generator().manual_seed(1_000_003 * int(seed) + salt)
    kv = torch.randint(1, 5, (4, 3), generator=g).tolist()
    amp = torch.randn(4, generator=g, dtype=torch.float64).tolist()
    phi = (2 * math.pi * torch.rand(4, generator=g, dtype=torch.float64)).tolist()
    x, y, z = ((torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n for n in (ni, nj, nk))
    gd = torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)
    q = 1e-3 * (2 * torch.rand((nk, nj, ni), generator=gd, device="cuda", dtype=torch.float64) - 1)
    for (kx, ky, kz), a, p in zip(kv, amp, phi):
        arg = (kx * x)[None, None, :] + (ky * y)[None, :, None] + (kz * z)[:, None, None]
        q += a * torch.sin(2 * math.pi * arg + p)
    return q


def _specs(case, seed):
    """The instances of a batch: grids and slice counts from "mix", parameters and fields from the seed."""
    r = random.Random(case["mix"])
    out = []
    for i in range(case["instances"]):
        n, slices = r.choice(BATCH_SIZES), r.randint(8, 16)
        s = random.Random(1000 * int(seed) + i)
        out.append(dict(case, kind="parareal", n=n, slices=slices, nu=10 ** s.uniform(-4, -2), cx=s.uniform(-1, 1),
                        cy=s.uniform(-1, 1), cz=s.uniform(-1, 1), g="rk4", gprec="f32"))
    return out


def _steps_of(c):
    """(fine step, coarse step, end time) of a Parareal case."""
    dtc = _dt(c, c["n"], coarse=True)
    dtf = min(dtc * c["coarse"] / c["fine"], _dt(c, c["n"]))
    end = dtf * c["fine"] * c["slices"]
    return end / (c["fine"] * c["slices"]), end / (c["coarse"] * c["slices"]), end


def _conv(c, ni, nj, nk):
    return sp.Convection(ni, nj, nk, 1.0 / ni, c["nu"], c["nufreq"], c["cx"], c["cy"], c["cz"], upwind=c["upwind"],
                         device=DEVICE)


def _parareal(c, seed, salt=0):
    n = c["n"]
    conv = _conv(c, n, n, n)
    if c["tune"] == "pairs":
        conv.set_tune(sp.SP_F64, c["slices"], 16, 64, 4)
    _, _, end = _steps_of(c)
    conf = sp.RuntimeConfiguration(timeSlices=c["slices"], nu0=c["nu"], nufreq=c["nufreq"], cx=c["cx"], cy=c["cy"],
                                   cz=c["cz"], gridSize=n, endTime=end, timeStepsFine=c["fine"] * c["slices"],
                                   timeStepsCoarse=c["coarse"] * c["slices"], kmax=c["kmax"])
    q0, q = conv.field(), conv.field()
    conv.upload(q0, _field(seed, salt, n, n, n))
    return sp.Parareal(conv, q0, q, 0.0, conf, coarse=c["g"], coarse_precision=c["gprec"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "parareal":
        return dict(case=case, par=_parareal(case, seed))
    if kind == "batch":
        pars = [_parareal(s, seed, i) for i, s in enumerate(_specs(case, seed))]
        return dict(case=case, pars=pars, batch=PararealBatch(pars))
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    dt = _dt(case, ni)
    q0 = _field(seed, 0, nk, nj, ni)
    if kind == "autograd":
        p = torch.tensor([case["nu"], case["cx"], case["cy"], case["cz"]], dtype=torch.float64)
        return dict(case=case, dt=dt, q0=q0.requires_grad_(), params=p.requires_grad_(),
                    weight=_field(seed, 1, nk, nj, ni))
    conv = _conv(case, ni, nj, nk)
    if kind == "host":
        host = torch.empty((nk, nj, ni), dtype=torch.float64, pin_memory=True)
        host.copy_(q0)
        return dict(case=case, dt=dt, conv=conv, host=host.numpy())
    prec = sp.SP_F64 if case["prec"] == "f64" else sp.SP_F32
    if case["tune"] == "pairs":
        conv.set_tune(sp.SP_F64, 1, 16, 64 if nk >= 64 else 0, 4)
    a, b = conv.field(prec), conv.field(prec)
    conv.upload(a, q0)
    s = dict(case=case, dt=dt, conv=conv, a=a, b=b)
    if kind == "gradient" or case.get("errors"):
        s["ref"] = conv.field()
        conv.upload(s["ref"], _field(seed, 1, nk, nj, ni))
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "parareal":
        rep = state["par"].DoParallel()
        return {"q": state["par"].solution.interior(), "iterations": rep["iterations"]}
    if kind == "batch":
        reps, _ = state["batch"].run()
        return {"q": [p.solution.interior() for p in state["pars"]], "iterations": [r["iterations"] for r in reps]}
    if kind == "autograd":
        q0, params = state["q0"], state["params"]
        q = rk4_propagate(q0, params, 1.0 / case["ni"], 0.0, state["dt"], case["steps"],
                          checkpoint_every=case["every"], nufreq=case["nufreq"], upwind=case["upwind"])
        gq, gp = torch.autograd.grad((q * state["weight"]).sum(), (q0, params))
        return {"q": q.detach(), "grad_q0": gq, "grad_params": gp}
    conv = state["conv"]
    if kind == "host":
        return {"q": conv.DoRK4Host(state["host"], 0.0, state["dt"], case["steps"])}
    if kind == "gradient":
        j, grad, gp = misfit_gradient(conv, state["a"], state["ref"], 0.0, state["dt"], case["steps"],
                                      checkpoint_every=case["every"])
        return {"J": j, "grad_q0": grad.interior(), "grad_params": gp}
    if kind == "euler":
        conv.DoEuler(state["a"], state["b"], 0.0, state["dt"], case["steps"])
    elif case["steps"] == 1:
        conv.DoRK4Timestep(state["a"], state["b"], 0.0, state["dt"])
    else:
        conv.DoRK4(state["a"], state["b"], 0.0, state["dt"], case["steps"])
    out = {"q": state["b"].interior()}
    if case["errors"]:
        out["err_max"], out["err_l2"] = conv.errors(state["b"], state["ref"])
    return out


# ---------------------------------------------------------------------------
# Work and exact values.

RK4_FLOPS = 4 * 27 + 12   # 13-point sums of the four stages and their updates, per cell and step
EULER_FLOPS = 18


def work(case):
    """Flops of the steps that the scheme prescribes; bytes of the inputs and outputs alone."""
    kind = case["kind"]
    if kind == "batch":
        parts = [work(s) for s in _specs(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "parareal":
        cells, p = case["n"] ** 3, case["slices"]
        g = RK4_FLOPS if case["g"] == "rk4" else EULER_FLOPS
        fine = sum(p - k for k in range(case["kmax"])) * case["fine"]
        coarse = (p + sum(p - k for k in range(case["kmax"]))) * case["coarse"]
        return {"bytes": 16.0 * cells, "flops": float(cells * (fine * RK4_FLOPS + coarse * g))}
    cells = case["ni"] * case["nj"] * case["nk"]
    es = 4 if case["prec"] == "f32" else 8
    if kind in ("gradient", "autograd"):
        # one forward run and the adjoint of every stage with its four parameter sums
        return {"bytes": 24.0 * cells, "flops": float(cells * case["steps"] * (RK4_FLOPS + 4 * 40))}
    per = EULER_FLOPS if kind == "euler" else RK4_FLOPS
    return {"bytes": 2.0 * cells * es + (16.0 * cells if case.get("errors") else 0.0),
            "flops": float(cells * case["steps"] * per)}


def _nu(nu0, nufreq, t):
    return nu0 * (1.0 + 0.5 * math.sin(nufreq * t))


def _rhs4(q, dx, nu, c):
    """Fourth-order central advection and Laplacian on the periodic box, axes (..., z, y, x)."""
    r = (-90.0 * nu / (12 * dx * dx)) * q
    for d, cd in zip((-1, -2, -3), c):
        m1, p1, m2, p2 = (torch.roll(q, s, d) for s in (1, -1, 2, -2))
        r = r + cd / (12 * dx) * (8 * (m1 - p1) - (m2 - p2)) + nu / (12 * dx * dx) * (16 * (m1 + p1) - (m2 + p2))
    return r


def _rhs2(q, dx, nu, c, upwind):
    r = (-6.0 * nu / (dx * dx)) * q
    for d, cd in zip((-1, -2, -3), c):
        m1, p1 = torch.roll(q, 1, d), torch.roll(q, -1, d)
        adv = (-cd / dx) * ((q - m1) if cd > 0 else (p1 - q)) if upwind else cd / (2 * dx) * (m1 - p1)
        r = r + adv + nu / (dx * dx) * (m1 + p1)
    return r


def _rk4_step(q, dx, nu, c, dt):
    k1 = _rhs4(q, dx, nu, c)
    k2 = _rhs4(q + (0.5 * dt) * k1, dx, nu, c)
    k3 = _rhs4(q + (0.5 * dt) * k2, dx, nu, c)
    k4 = _rhs4(q + dt * k3, dx, nu, c)
    return q + (dt / 6) * (k1 + 2 * k2 + 2 * k3 + k4)


def _propagate(q, case, dx, t0, dt, n, euler):
    c = (case["cx"], case["cy"], case["cz"])
    for i in range(n):
        nu = _nu(case["nu"], case["nufreq"], t0 + i * dt)
        q = q + dt * _rhs2(q, dx, nu, c, case["upwind"]) if euler else _rk4_step(q, dx, nu, c, dt)
    return q


def _exact_parareal(case, seed, salt=0):
    n, p, euler = case["n"], case["slices"], case["g"] == "euler"
    dx, c = 1.0 / n, (case["cx"], case["cy"], case["cz"])
    dtf, dtc, end = _steps_of(case)
    size = end / p

    def coarse(q, t0, steps):
        return _propagate(q, case, dx, t0, dtc, steps, euler)

    # predictor from t = 0 for every slice, then G of each slice's own start
    u = [_field(seed, salt, n, n, n)]
    for r in range(1, p):
        u.append(coarse(u[-1], (r - 1) * case["coarse"] * dtc, case["coarse"]))
    gold = [coarse(u[r], size * r, case["coarse"]) for r in range(p)]
    u.append(gold[-1])
    for _ in range(case["kmax"]):
        f = torch.stack(u[:p])
        for i in range(case["fine"]):
            nu = torch.tensor([_nu(case["nu"], case["nufreq"], size * r + i * dtf) for r in range(p)], device="cuda",
                              dtype=torch.float64)
            f = _rk4_step(f, dx, nu.view(-1, 1, 1, 1), c, dtf)
        new = [u[0]]
        for r in range(p):
            g = coarse(new[r], size * r, case["coarse"])
            new.append(g + f[r] - gold[r])
            gold[r] = g
        u = new
    return u[p]


def exact(case, seed):
    kind = case["kind"]
    if kind == "parareal":
        return {"q": _exact_parareal(case, seed), "iterations": None}
    if kind == "batch":
        specs = _specs(case, seed)
        return {"q": [_exact_parareal(s, seed, i) for i, s in enumerate(specs)], "iterations": [None] * len(specs)}
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    dx, dt, n = 1.0 / ni, _dt(case, ni), case["steps"]
    q = _field(seed, 0, nk, nj, ni)
    if kind in ("gradient", "autograd"):
        return _exact_gradient(case, seed, q, dx, dt, n)
    if case["prec"] == "f32":
        q = q.float().double()
    q = _propagate(q, case, dx, 0.0, dt, n, kind == "euler")
    if kind == "host":
        return {"q": q}
    out = {"q": q}
    if case["errors"]:
        ref = _field(seed, 1, nk, nj, ni)
        out["err_max"] = float((q - ref).abs().max() / q.abs().max())
        out["err_l2"] = float((q - ref).norm() / ref.norm())
    return out


def _exact_gradient(case, seed, q, dx, dt, n):
    states = []
    params = torch.tensor([case["nu"], case["cx"], case["cy"], case["cz"]], dtype=torch.float64, device="cuda")

    def step(q, p, i):
        return _rk4_step(q, dx, p[0] * (1.0 + 0.5 * math.sin(case["nufreq"] * i * dt)), (p[1], p[2], p[3]), dt)

    for i in range(n):
        states.append(q)
        q = step(q, params, i)
    w = _field(seed, 1, case["nk"], case["nj"], case["ni"])
    lam = w if case["kind"] == "autograd" else q - w
    j = 0.5 * float((lam * lam).sum())
    gp = torch.zeros(4, dtype=torch.float64, device="cuda")
    for i in reversed(range(n)):
        with torch.enable_grad():
            qi, pi = states[i].requires_grad_(), params.clone().requires_grad_()
            lam, g = torch.autograd.grad(step(qi, pi, i), (qi, pi), lam)
        gp += g
    if case["kind"] == "autograd":
        return {"q": q, "grad_q0": lam, "grad_params": gp}
    return {"J": j, "grad_q0": lam, "grad_params": [float(v) for v in gp]}
