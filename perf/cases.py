"""The calls that a user of the step library makes, as cases to be timed.

Four ways into the library are covered, over the range of sizes that its
configurations, tests and benchmark use:

* ``stepper``: ``Stepper`` on one solve, 1D to 3D, plain FP64 or
  FP32-compensated.  A pass puts an initial field into the stepper and runs a
  number of steps, as a sweep over initial conditions does.
* ``save``: the same, ended by ``step_save``, the save step of the driver's
  main loop.
* ``batch``: ``BatchStepper`` on many uneven 1D and 2D solves.  A pass advances
  the batch and reads every solve's field.
* ``dropin``: one step of the reference's own loop through the functions of
  ``solver``, on CUDA tensors or on numpy arrays.

A field is ``early`` (the initial condition: X0 with white fluctuations) or
``developed`` (two phases with interfaces between them, which spread over many
table cells; a small share of the points lies outside the table's linear
region and takes the nearest-row fallback).
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from phasefield5d_b200 import workload as W
from phasefield5d_b200.batch import BatchStepper
from phasefield5d_b200.solver import elastic_setup
from phasefield5d_b200.solver import system as sysm
from phasefield5d_b200.solver.elastic import make_elastic_updater
from phasefield5d_b200.solver.fluxes import get_divergence_from_mu_function
from phasefield5d_b200.solver.interpolation import interpolator_nb
from phasefield5d_b200.solver.operators import (abs_max, calculate_laplacian, clamp_simplex,
                                                out_of_bounds)
from phasefield5d_b200.stepper import (Stepper, device_table, device_table32, reference_mu)

DEVICE = "cuda"
#: Phase contrast of a developed field, as a share of X0 per component, and
#: the largest change of their sum (the linear region ends near 1).
CONTRAST, CONTRAST_SUM = (-0.4, 0.4, -0.3, 0.7), 0.085
#: (temperature, Omega seed, composition) of the solves of a batch: four
#: temperature tables, compositions inside the spinodal of each.
BATCH_1D = ((773.0, 0, (0.364, 0.073, 0.175, 0.094)), (973.0, 4, (0.176, 0.053, 0.179, 0.141)),
            (773.0, 0, (0.400, 0.055, 0.079, 0.145)), (973.0, 4, (0.071, 0.175, 0.306, 0.160)))
BATCH_2D = ((873.0, 1, (0.095, 0.137, 0.133, 0.283)), (1073.0, 215, (0.151, 0.134, 0.197, 0.104)),
            (873.0, 1, (0.065, 0.063, 0.207, 0.312)), (1073.0, 215, (0.101, 0.071, 0.230, 0.157)))


def listed():
    return [
        # the driver near a save time: single steps of a small 1D solve, read back each time
        stepper("1d_203_fp64_1step", (203,), "fp64", 1),
        # the 1D workload of the benchmark (fixed dt), run for a while
        stepper("1d_1280_fp64", (1280,), "fp64", 200, adaptive=False),
        # a long 1D solve of the precision form, sides as in the batched workload
        stepper("1d_4112_fp32c", (4112,), "fp32c", 100),
        # the headline workload
        stepper("2d_512_fp64", (512, 512), "fp64", 20),
        # a ragged 2D field late in a run
        stepper("2d_389x250_fp64_developed", (389, 250), "fp64", 20, field="developed"),
        # the headline workload in the precision form, late in a run
        stepper("2d_512_fp32c", (512, 512), "fp32c", 20, field="developed"),
        # the 3D workload of the benchmark in its two forms: the largest fields
        stepper("3d_256_fp64", (256, 256, 256), "fp64", 4, resolution=0.02),
        stepper("3d_256_fp32c", (256, 256, 256), "fp32c", 8, resolution=0.02),
        # a ragged 3D field late in a run, closed by a save step
        stepper("3d_97x75x130_fp64_save", (97, 75, 130), "fp64", 6, field="developed", way="save"),
        # the batched workload of the benchmark: 64 uneven solves
        {"name": "batch_64", "way": "batch", "solves": 64, "steps": 50, "shapes": 2026,
         "field": "early"},
        # the reference's loop body with its arrays kept on the GPU
        dropin("dropin_3d_128_cuda", (128, 128, 128), "cuda"),
        # the reference's loop body unchanged, on its numpy arrays
        dropin("dropin_2d_200x160_numpy", (200, 160), "numpy"),
    ]


def stepper(name, shape, precision, steps, *, way="stepper", field="early", resolution=0.025,
            elastic=True, adaptive=True):
    case = {"way": way, "dim": len(shape), "n0": shape[0], "n1": shape[1] if len(shape) > 1 else 1,
            "n2": shape[2] if len(shape) > 2 else 1, "precision": precision, "steps": steps,
            "field": field, "resolution": resolution, "elastic": elastic, "adaptive": adaptive}
    return {"name": name, **case} if name else case


def dropin(name, shape, arrays, *, field="early", elastic=True):
    case = {"way": "dropin", "dim": len(shape), "n0": shape[0],
            "n1": shape[1] if len(shape) > 1 else 1, "n2": shape[2] if len(shape) > 2 else 1,
            "arrays": arrays, "field": field, "resolution": 0.025, "elastic": elastic}
    return {"name": name, **case} if name else case


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def shape_of(dim, scale=1.0):
        if dim == 1:
            return (side(64, 8192),)
        if dim == 2:
            return (side(24, 900 * scale), side(24, 900 * scale))
        return tuple(side(16, 220 * scale) for _ in range(3))

    way = rng.choice(["stepper", "stepper", "stepper", "stepper", "save", "batch", "dropin",
                      "dropin"])
    field = rng.choice(["early", "developed"])
    if way == "batch":
        return {"way": "batch", "solves": side(2, 64), "steps": rng.choice([10, 25, 50]),
                "shapes": rng.randrange(1 << 30), "field": field}
    dim = rng.choice([1, 2, 2, 3, 3])
    if way == "dropin":
        arrays = rng.choice(["cuda", "cuda", "numpy"])
        return dropin(None, shape_of(dim, 0.6 if arrays == "cuda" else 0.3), arrays, field=field,
                      elastic=rng.random() < 0.8)
    shape = shape_of(dim)
    if dim >= 2 and rng.random() < 0.3:          # the sides that ppw and mw give: powers of two
        shape = (rng.choice([64, 128, 256, 512]),) * 2 if dim == 2 else (rng.choice([32, 64, 128]),) * 3
    points = math.prod(shape)
    steps = max(1, min(rng.choice([1, 5, 20, 50]), 30_000_000 // points))
    return stepper(None, shape, rng.choice(["fp64", "fp64", "fp32c"]), steps, way=way, field=field,
                   resolution=rng.choice([0.025, 0.025, 0.02]), elastic=rng.random() < 0.85,
                   adaptive=rng.random() < 0.8)


# ---------------------------------------------------------------------------
# What a program keeps between solves: tables and scalars of an alloy
# ---------------------------------------------------------------------------

def shape_of_case(case):
    return (case["n0"], case["n1"], case["n2"])[:case["dim"]]


@functools.lru_cache(maxsize=None)
def alloy(dim, resolution):
    """Host setup (table, CTLD scan, dx, dt) of the named workload of a dimension."""
    cfg = {1: W.config_1d_fixed, 2: W.config_2d_adaptive, 3: W.config_3d_precision}[dim]()
    cfg.resolution, cfg.omega_seed, cfg.n_k, cfg.shape = resolution, 4, 2000, (16,) * dim
    return W.build_problem(cfg)


@functools.lru_cache(maxsize=None)
def batch_alloy(dim, which):
    temperature, seed, x0 = (BATCH_1D, BATCH_2D)[dim - 1][which]
    cfg = W.SolveConfig(system_dim=dim, initial_composition=x0, kappa_value=1e-15, n_k=500,
                        temperature=temperature, shape=(16,) * dim)
    return W.build_problem(cfg, table=batch_table(temperature, seed))


@functools.lru_cache(maxsize=None)
def batch_table(temperature, seed):
    return W.make_table(0.025, temperature, seed)


BATCH_TABLES = {}


@functools.lru_cache(maxsize=None)
def table_of(dim, resolution, precision):
    prob = alloy(dim, resolution)
    if precision == "fp64":
        return device_table(prob.grid, torch), None
    mu0 = reference_mu(prob.grid, resolution, prob.X0)
    return device_table32(prob.grid, mu0, torch), mu0


@functools.lru_cache(maxsize=64)
def bk_of(shape, dx):
    k_grid, k_norm = sysm.build_fourier_grid_for(len(shape), shape, dx, (1, 0, 0))
    return np.ascontiguousarray(elastic_setup.build_khachaturyan_kernel(k_grid, k_norm, 240.0,
                                                                        150.0, 120.0))


def smooth(shape, gen):
    """A periodic random field, normalised, with structure at about 16 cells."""
    white = torch.randn(shape, dtype=torch.float64, device=DEVICE, generator=gen)
    q2 = 0.0
    for d, n in enumerate(shape):
        f = torch.fft.fftfreq(n, device=DEVICE, dtype=torch.float64) if d < len(shape) - 1 else \
            torch.fft.rfftfreq(n, device=DEVICE, dtype=torch.float64)
        q2 = q2 + (f ** 2).reshape([-1 if e == d else 1 for e in range(len(shape))])
    spec = torch.fft.rfftn(white) * torch.exp(-(16.0 * q2.sqrt() - 1.0) ** 2 * 4.0)
    out = torch.fft.irfftn(spec, s=shape)
    return out / out.std().clamp_min(1e-30)


def field_of(shape, x0, kind, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    base = torch.as_tensor(x0, dtype=torch.float64, device=DEVICE)
    noise = torch.rand((*shape, 5), dtype=torch.float64, device=DEVICE, generator=gen) * 2.0 - 1.0
    noise -= noise.mean(dim=-1, keepdim=True)
    X = base + 1e-3 * noise[..., 1:]
    del noise
    if kind == "developed":
        phase = torch.tanh(2.0 * smooth(shape, gen))
        share = min(1.0, CONTRAST_SUM / abs(sum(x * k for x, k in zip(x0, CONTRAST))))
        for c in range(4):
            X[..., c] += share * x0[c] * CONTRAST[c] * phase
            X[..., c] += 0.04 * x0[c] * smooth(shape, gen)
    return X.contiguous()


def stepper_args(case):
    shape = shape_of_case(case)
    prob = alloy(case["dim"], case["resolution"])
    adaptive = case["adaptive"]
    return prob, shape, dict(
        grid=prob.grid, resolution=case["resolution"], node_coord=prob.node_coord, X0=prob.X0,
        kappa=prob.kappa, dx=prob.dx, lvec=prob.lvec if case["elastic"] else None,
        bk=bk_of(shape, prob.dx) if case["elastic"] else None, ctld=prob.ctld, t_cfl=prob.t_cfl,
        dt=prob.dt0 if adaptive else min(prob.dt0, prob.t_cfl), adaptive=adaptive,
        lower_limit=prob.cfg.lower_limit, upper_limit=prob.cfg.upper_limit)


def batch_members(case):
    """(alloy, shape) of each solve: alternately 1D (2048 to 8192 points) and
    2D (128 to 384 cells a side), as the benchmark's batched workload."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for i in range(case["solves"]):
        if i % 2 == 0:
            out.append((batch_alloy(1, (i // 2) % 4), (int(rng.choice(np.arange(2048, 8193, 16))),)))
        else:
            n = int(rng.choice(np.arange(128, 385, 16)))
            out.append((batch_alloy(2, (i // 2) % 4), (n, n)))
    return out


def batch_fields(case, seed):
    return [field_of(shape, prob.X0, case["field"], 1000 * seed + i)
            for i, (prob, shape) in enumerate(batch_members(case))]


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    if case["way"] == "batch":
        probs = [dataclasses.replace(prob, shape=shape, bk=bk_of(shape, prob.dx),
                                     X_init=X.cpu().numpy())
                 for (prob, shape), X in zip(batch_members(case), batch_fields(case, seed))]
        return {"case": case, "batch": BatchStepper(probs, table_cache=BATCH_TABLES)}
    shape = shape_of_case(case)
    if case["way"] == "dropin":
        prob = alloy(case["dim"], case["resolution"])
        X = field_of(shape, prob.X0, case["field"], seed)
        empty = functools.partial(torch.empty, dtype=torch.float64, device=DEVICE)
        state = {"X0": X, "X": empty((*shape, 4)), "dX": empty((*shape, 4)),
                 "lap": empty((*shape, 4)), "interp": empty((*shape, 9)),
                 "mask": torch.empty(shape, dtype=torch.bool, device=DEVICE)}
        if case["arrays"] == "numpy":
            state = {k: v.cpu().numpy() for k, v in state.items()}
        cfg = dataclasses.replace(prob.cfg, include_cubic_anisotropy=case["elastic"])
        elastic = make_elastic_updater(cfg, prob.Lambda, bk_of(shape, prob.dx), (*shape, 4))
        kappa = prob.kappa if case["arrays"] == "numpy" else torch.from_numpy(prob.kappa).to(DEVICE)
        return {"case": case, "prob": prob, "elastic": elastic, "kappa": kappa,
                "div": get_divergence_from_mu_function(case["dim"]), **state}
    prob, shape, args = stepper_args(case)
    table, mu0 = table_of(case["dim"], case["resolution"], case["precision"])
    X = field_of(shape, prob.X0, case["field"], seed)
    st = Stepper(X=X, precision=case["precision"], table=table, table_mu0=mu0, **args)
    return {"case": case, "X": X, "stepper": st, "dt": args["dt"]}


def run(state):
    way = state["case"]["way"]
    if way == "batch":
        b = state["batch"]
        b.advance(state["case"]["steps"])
        return {"fields": [b.field(i) for i in range(len(b.problems))]}
    if way == "dropin":
        return run_dropin(state)
    st = state["stepper"]
    st.X.copy_(state["X"])
    st.reset(state["dt"])
    fp64 = state["case"]["precision"] == "fp64"
    if way == "save":
        s = st.run(state["case"]["steps"] - 1) if state["case"]["steps"] > 1 else None
        d = st.step_save()
        # net and total_flux are left out: sums that cancel, of which only rounding is left
        out = {k: d[k] for k in ("mass", "comp_min", "comp_max", "comp_fe_min", "comp_var")}
        if fp64:
            out.update({k: d[k] for k in ("max_change", "f_grad", "xdotmax", "dt", "time")})
        halted = d["halted"] or bool(s and s["halted"])
    else:
        s = st.run(state["case"]["steps"])
        out = {"dt": s["dt"], "time": s["time"]} if fp64 else {}
        halted = s["halted"]
    out.update(field=st.field(), halted=halted)
    if fp64:
        out["rate"] = st.rate().clone()      # rate() is a view of the stepper's buffer
    return out


def run_dropin(s):
    """The loop body of the reference (examples/simulate.py:242-320)."""
    prob, X, dX = s["prob"], s["X"], s["dX"]
    if isinstance(X, np.ndarray):
        X[...] = s["X0"]
    else:
        X.copy_(s["X0"])
    out_of_bounds(X)
    interp = interpolator_nb(X, prob.grid, prob.cfg.resolution, prob.tree, prob.calphad_values,
                             out=s["interp"], mask_buffer=s["mask"])
    mu, M = interp[..., :4], interp[..., 4:]
    lap = calculate_laplacian(X, prob.dx, out=s["lap"])
    lap *= s["kappa"]
    mu -= lap
    s["elastic"](mu, X)
    s["div"](X, M, mu, 1.0 / prob.dx, dX)
    xdotmax = abs_max(dX)
    dt = sysm.apply_adaptive_time(prob.dt0, xdotmax, prob.ctld, prob.t_cfl)
    dX *= dt
    X += dX
    clamp_simplex(X)
    return {"X": X, "dX": dX, "interp": s["interp"], "mask": s["mask"], "xdotmax": xdotmax,
            "dt": dt}


def work(case):
    """Bytes and operations of a pass.  A step of one point reads and writes
    its composition and its rate and takes its misfit through the transform
    pair (FP64 176 bytes, precision form 120); about 650 operations."""
    if case["way"] == "batch":
        points = sum(math.prod(shape) for _, shape in batch_members(case))
        return {"bytes": (120.0 * case["steps"] + 48) * points, "flops": 650.0 * case["steps"] * points}
    points = math.prod(shape_of_case(case))
    if case["way"] == "dropin":
        # X twice over each of the eight calls' inputs and outputs
        return {"bytes": 660.0 * points, "flops": 650.0 * points}
    step = 176.0 if case["precision"] == "fp64" else 120.0
    if not case["elastic"]:
        step -= 48.0 if case["precision"] == "fp64" else 24.0
    return {"bytes": (step * case["steps"] + 96) * points, "flops": 650.0 * case["steps"] * points}


# ---------------------------------------------------------------------------
# exact: the same step in plain torch, 64 bits
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def plain_table(key):
    prob = batch_alloy(*key[1:]) if key[0] == "batch" else alloy(*key[1:])
    rows = torch.from_numpy(np.ascontiguousarray(prob.table.data)).to(DEVICE)
    return torch.from_numpy(prob.grid).to(DEVICE).reshape(-1, 9), rows[rows[:, :4].sum(1) > 0.6]


def plain_interp(X, resolution, n, grid, rows):
    shape = X.shape[:-1]
    x = X.reshape(-1, 4)
    u = x * (1.0 / resolution)
    i = u.floor().clamp(0, n - 2)
    t = (u - i).clamp(0.0, 1.0)
    i = i.to(torch.int64)
    out = torch.zeros((x.shape[0], 9), dtype=torch.float64, device=DEVICE)
    for c in range(16):
        node, w = 0, 1.0
        for d in range(4):
            b = (c >> (3 - d)) & 1
            node = node * n + i[:, d] + b
            w = w * (t[:, d] if b else 1.0 - t[:, d])
        out += w[:, None] * grid[node]
    linear = x[:, 0] + x[:, 1] + x[:, 2] + x[:, 3] <= 1.0 - 4.0 * resolution - 1e-9
    far = (~linear).nonzero()[:, 0]
    for part in far.split(1024):
        d2 = sum((x[part, d, None] - rows[None, :, d]) ** 2 for d in range(4))
        out[part] = rows[d2.argmin(1), 4:]
    return out.reshape(*shape, 9), linear.reshape(shape)


def plain_rate(X, a, table):
    """(table values, linear mask, mu, dX/dt) of a field; a: the solve's numbers."""
    dims = range(X.dim() - 1)
    v, linear = plain_interp(X, a["resolution"], a["n"], *table)
    lap = -2.0 * len(dims) * X
    for d in dims:
        lap += torch.roll(X, -1, d)
        lap += torch.roll(X, 1, d)
    lap *= 1.0 / (a["dx"] * a["dx"])
    mu = v[..., :4] - lap * a["kappa"]
    del lap
    if a["bk"] is not None:
        s = ((X - a["x0"]) * a["l"]).sum(-1)
        s = torch.fft.irfftn(torch.fft.rfftn(s) * a["bk"], s=s.shape)
        mu += s[..., None] * a["l"]
    M = v[..., 4:]
    rate = torch.zeros_like(X)
    for d in dims:
        xm = 0.5 * (X + torch.roll(X, -1, d))
        mm = 0.5 * (M + torch.roll(M, -1, d))
        g = (torch.roll(mu, -1, d) - mu) * (1.0 / a["dx"])
        fe = (1.0 - xm.sum(-1, keepdim=True)) * mm[..., :1]
        dot = (xm * g).sum(-1, keepdim=True)
        wk = xm * mm[..., 1:] * (g - dot)
        J = xm * (fe * dot - wk.sum(-1, keepdim=True)) + wk
        rate += J
        rate -= torch.roll(J, 1, d)
    return v, linear, mu, rate * (1.0 / a["dx"])


def plain_dt(dt, xdotmax, a):
    raw = dt
    if xdotmax > 0.0:
        raw = min(max(dt, a["lower"] / xdotmax), a["upper"] / xdotmax)
    return min(2.0 * dt, raw, 0.005 * a["ctld"], a["t_cfl"])


def plain_update(X, dX):
    X = X + dX
    return X / X.sum(-1, keepdim=True).clamp_min(1.0)


def plain_args(prob, shape, resolution, elastic):
    dev = functools.partial(torch.as_tensor, dtype=torch.float64, device=DEVICE)
    return {"resolution": resolution, "n": prob.grid.shape[0], "dx": prob.dx,
            "kappa": dev(prob.kappa), "x0": dev(prob.X0), "ctld": prob.ctld, "t_cfl": prob.t_cfl,
            "lower": prob.cfg.lower_limit, "upper": prob.cfg.upper_limit,
            "bk": dev(bk_of(shape, prob.dx)) if elastic else None,
            "l": dev(prob.lvec) if elastic else None}


def plain_steps(X, a, table, dt, steps, adaptive):
    time = 0.0
    for _ in range(steps):
        before = X
        mu, rate = plain_rate(X, a, table)[2:]
        if adaptive:
            dt = plain_dt(dt, float(rate.abs().max()), a)
        time += dt
        X = plain_update(X, rate * dt)
    return before, mu, rate, X, dt, time


def exact(case, seed):
    if case["way"] == "batch":
        fields = []
        members = batch_members(case)
        for i, ((prob, shape), X) in enumerate(zip(members, batch_fields(case, seed))):
            table = plain_table(("batch", len(shape), (i // 2) % 4))
            a = plain_args(prob, shape, 0.025, True)
            fields.append(plain_steps(X, a, table, prob.dt0, case["steps"], True)[3])
        return {"fields": fields}
    shape = shape_of_case(case)
    prob = alloy(case["dim"], case["resolution"])
    table = plain_table(("alloy", case["dim"], case["resolution"]))
    a = plain_args(prob, shape, case["resolution"], case["elastic"])
    X = field_of(shape, prob.X0, case["field"], seed)
    if case["way"] == "dropin":
        v, linear, mu, rate = plain_rate(X, a, table)
        v[..., :4] = mu
        xdotmax = float(rate.abs().max())
        dt = plain_dt(prob.dt0, xdotmax, {**a, "lower": 1e-5, "upper": 1e-3})
        return {"X": plain_update(X, rate * dt), "dX": rate * dt, "interp": v, "mask": linear,
                "xdotmax": xdotmax, "dt": dt}
    dt0 = prob.dt0 if case["adaptive"] else min(prob.dt0, prob.t_cfl)
    before, mu, rate, X, dt, time = plain_steps(X, a, table, dt0, case["steps"], case["adaptive"])
    out = {"field": X, "halted": False}
    fp64 = case["precision"] == "fp64"
    if fp64:
        out.update(dt=dt, time=time, rate=rate)
    if case["way"] == "save":
        flat = X.reshape(-1, 4)
        lap = -2.0 * case["dim"] * X
        for d in range(case["dim"]):
            lap = lap + torch.roll(X, -1, d) + torch.roll(X, 1, d)
        lap /= prob.dx ** 2
        out.update(mass=flat.sum(0), comp_min=flat.amin(0), comp_max=flat.amax(0),
                   comp_fe_min=float(1.0 - flat.sum(1).max()),
                   comp_var=flat.var(0, unbiased=False))
        if fp64:
            out.update(max_change=rate.abs().reshape(-1, 4).amax(0), xdotmax=float(rate.abs().max()),
                       f_grad=float(-0.5 * prob.dx ** case["dim"] * (X * a["kappa"] * lap).sum()))
    return out
