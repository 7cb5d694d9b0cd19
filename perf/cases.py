"""The measured workloads of the reacting-Euler step: what a program that uses this
framework has it do, over the sizes it is used at.

Kinds (the "kind" of a case):
  eos       properties(): p, a, T of a batch of cells (diagnostics, inflow set-up, tagging)
  flow      one flow(h) of a one-patch level as a host program drives it call by call:
            cfl_dt, ghost fill, Euler stage, ghost fill, Euler stage with Heun combine
  chem      ChemistryBatch.advance: the chemistry of a Strang step for a batch of cells
  ignition  ChemSensitivity.adjoint: ignition delay (or final T) of 0D cells and its
            gradient in the 21 log rate constants
  strang    Stepper: state in from pinned host memory, Strang steps, state out
  amr       AmrStepper: Strang steps on a three-level hierarchy, one regrid
  adjoint   FlowAdjoint: a recorded run and its reverse sweep

Everything is double precision, as the framework is.  The species and reaction numbers that
exact() needs come from the mechanism file's fixture; its arithmetic is written out here.
"""
import json
import math
import os

import numpy as np
import torch

ATM = 101325.0
RU = 8314.46261815324
NAMES = ["H2", "O2", "H2O", "H", "O", "OH", "HO2", "H2O2", "N2", "AR"]
ATOMS = {"H": 1.008, "O": 15.999, "N": 14.007}


def listed():
    return [
        # the cells of the 2000 x 2 planar detonation: a call that launches and little else
        dict(name="eos_line", kind="eos", cells=4000, ns=10),
        # every cell of the 2048 x 512 cellular detonation
        dict(name="eos_grid", kind="eos", cells=2048 * 512, ns=10),
        # flow(dt/2) of the 2048 x 512 detonation level, per-face kernels, periodic in y
        dict(name="flow_det2d", kind="flow", nx=2048, ny=512, ns=10, form="plain", wedge=False),
        # flow(dt/2) of the oblique detonation over a wedge at the Teng case's finest level,
        # the fused kernel, inflow and wedge boundaries
        dict(name="flow_wedge", kind="flow", nx=576, ny=256, ns=9, form="fused", wedge=True),
        # the chemistry-only batch of very uneven stiffness, own interval per cell
        dict(name="chem_uneven", kind="chem", cells=1 << 16, ns=10, form="batched", field="uneven"),
        # react(dt) on a level crossed by a detonation: fresh, igniting and burnt cells
        dict(name="chem_front", kind="chem", cells=512 * 128, ns=10, form="batched", field="front"),
        # the drop-in form (one thread per cell) on igniting H2/air cells
        dict(name="chem_drop_in", kind="chem", cells=3000, ns=9, form="plain", field="ignition"),
        # sensitivities of the heat-release time of a batch of 0D H2/air cells
        dict(name="ignition_adjoint", kind="ignition", cells=1024, ncalls=8, objective="ignition_delay"),
        # the headline run: the first Strang steps of the 2048 x 512 cellular detonation, whose
        # hot band ignites
        dict(name="strang_det2d", kind="strang", nx=2048, ny=512, ns=10, steps=2),
        # a developed planar detonation, 2000 x 2 cells, device-resident steps
        dict(name="strang_det1d", kind="strang", nx=2000, ny=2, ns=10, steps=8),
        # wedge on three levels of block AMR with one regrid
        dict(name="amr_wedge", kind="amr", nx=256, ny=128, steps=4),
        # induction-length sensitivities: a recorded 1D run and its adjoint
        dict(name="adjoint_det1d", kind="adjoint", nx=1000, ny=2, steps=2, chemistry=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eos", "flow", "flow", "chem", "chem", "chem", "ignition", "strang", "strang", "amr", "adjoint"])
    ns = rng.choice([9, 10])
    if kind == "eos":
        return dict(kind=kind, cells=_log(rng, 100, 1 << 20), ns=ns)
    if kind == "flow":
        nx, ny = _log(rng, 24, 2048), _log(rng, 2, 512)
        return dict(kind=kind, nx=nx, ny=ny, ns=ns, form=rng.choice(["plain", "fused"]), wedge=rng.random() < 0.4)
    if kind == "chem":
        field = rng.choice(["uneven", "front", "ignition"])
        top = {"uneven": 1 << 15, "front": 1 << 16, "ignition": 1 << 14}[field]
        return dict(kind=kind, cells=_log(rng, 64, top), ns=ns, form=rng.choice(["batched", "batched", "plain"]),
                    field=field)
    if kind == "ignition":
        return dict(kind=kind, cells=_log(rng, 32, 1024), ncalls=rng.randint(2, 8),
                    objective=rng.choice(["ignition_delay", "final_T"]))
    if kind == "strang":
        nx, ny = _log(rng, 96, 2048), _log(rng, 2, 512)
        return dict(kind=kind, nx=nx, ny=ny, ns=ns, steps=rng.randint(1, 2))
    if kind == "amr":
        return dict(kind=kind, nx=16 * rng.randint(4, 16), ny=16 * rng.randint(2, 8), steps=4)
    return dict(kind=kind, nx=_log(rng, 64, 1000), ny=rng.choice([2, 3]), steps=rng.randint(1, 2),
                chemistry=rng.random() < 0.5)


# ------------------------------------------------------------------ species data
def _fixture():
    if not hasattr(_fixture, "data"):
        with open(os.path.join("tests", "golden", "h2li_mechanism.json")) as f:
            _fixture.data = json.load(f)
    return _fixture.data


def _species(ns, device="cuda"):
    """W (ns,), NASA7 low and high (ns, 7); the tenth species is inert argon."""
    by = {s["name"]: s for s in _fixture()["species"]}
    W, lo, hi = [], [], []
    for n in NAMES[:ns]:
        if n == "AR":
            W.append(39.95)
            lo.append([2.5, 0, 0, 0, 0, -745.375, 4.366])
            hi.append(lo[-1])
        else:
            W.append(sum(ATOMS[a] * v for a, v in by[n]["composition"].items()))
            lo.append(by[n]["nasa7"][0])
            hi.append(by[n]["nasa7"][1])
    t = lambda v: torch.tensor(v, dtype=torch.float64, device=device)  # noqa: E731
    return t(W), t(lo), t(hi)


def _h_RT(T, ns):
    """h_k/(R T), (ns, n)."""
    _, lo, hi = _species(ns, T.device)
    a = torch.where((T <= 1000.0)[None, :, None], lo[:, None, :], hi[:, None, :])
    return (a[..., 0] + T * (a[..., 1] / 2 + T * (a[..., 2] / 3 + T * (a[..., 3] / 4 + T * a[..., 4] / 5)))
            + a[..., 5] / T)


def _cp_R(T, ns):
    _, lo, hi = _species(ns, T.device)
    a = torch.where((T <= 1000.0)[None, :, None], lo[:, None, :], hi[:, None, :])
    return a[..., 0] + T * (a[..., 1] + T * (a[..., 2] + T * (a[..., 3] + T * a[..., 4])))


def _conserved(T, p, X, u, v):
    """Conserved states (NS + 3, n) of primitive ones; X (ns, n) mole fractions."""
    ns = X.shape[0]
    W = _species(ns, T.device)[0][:, None]
    Y = X * W / (X * W).sum(0)
    rho = p / (RU * T * (Y / W).sum(0))
    e = RU * T * ((Y / W) * (_h_RT(T, ns) - 1.0)).sum(0)
    return torch.cat([rho * Y, (rho * u)[None], (rho * v)[None], (rho * (e + 0.5 * (u * u + v * v)))[None]])


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)


def _log_uniform(g, n, lo, hi):
    return torch.exp(_uniform(g, n, math.log(lo), math.log(hi)))


# mole fractions of stoichiometric H2/O2 with 70% diluent, unburnt and burnt near 2800 K
FRESH = dict(H2=0.2, O2=0.1, dil=0.7)
BURNT = dict(H2=0.025, O2=0.012, H2O=0.16, H=0.008, O=0.004, OH=0.016, HO2=2e-6, H2O2=2e-7, dil=0.775)


def _mole(of, ns):
    x = torch.zeros(ns, dtype=torch.float64, device="cuda")
    for k, v in of.items():
        x[ns - 1 if k == "dil" else NAMES.index(k)] += v
    return x / x.sum()


def _front(seed, nx, ny, ns, dx):
    """(NS + 3, ny, nx): a right-running detonation in the left third of a grid: burnt gas,
    a reaction zone with radicals, an induction zone of shocked unburnt gas, fresh gas; the
    front's position and the states vary from row to row and by 1% from cell to cell."""
    g = _gen(seed)
    y = torch.arange(ny, dtype=torch.float64, device="cuda")[:, None]
    x = (torch.arange(nx, dtype=torch.float64, device="cuda")[None, :] + 0.5)
    ph = 2 * math.pi * torch.rand(3, dtype=torch.float64, device="cuda", generator=g)
    amp = 0.02 * nx
    k = 2 * math.pi * y / ny
    xf = 0.3 * nx + amp * (torch.sin(2 * k + ph[0]) + 0.5 * torch.sin(5 * k + ph[1]) + 0.25 * torch.sin(9 * k + ph[2]))
    ind = max(4.0, 0.02 * nx) * (1.0 + 0.5 * torch.sin(3 * k + ph[1]))  # induction length in cells
    zone = max(3.0, 0.02 * nx)
    s = xf - x  # > 0: behind the shock
    behind = s > 0
    prog = torch.where(behind, 0.5 * (1.0 + torch.tanh((s - ind) / zone * 2.0 - 2.0)), torch.zeros_like(s))
    prog = torch.where(prog < 1e-3, torch.zeros_like(prog), prog)
    noise = 1.0 + 0.02 * (torch.rand(ny, nx, dtype=torch.float64, device="cuda", generator=g) - 0.5)
    T = torch.where(behind, 1450.0 + 1400.0 * prog, torch.full_like(s, 298.0)) * noise
    p = torch.where(behind, 25.0 - 9.0 * prog, torch.ones_like(s)) * ATM
    u = torch.where(behind, 900.0 - 400.0 * prog, torch.zeros_like(s))
    v = torch.where(behind, 40.0 * torch.sin(3 * k + ph[2]).expand(ny, nx), torch.zeros_like(s))
    X = _mole(FRESH, ns)[:, None] * (1 - prog.reshape(-1)) + _mole(BURNT, ns)[:, None] * prog.reshape(-1)
    return _conserved(T.reshape(-1), p.reshape(-1), X, u.reshape(-1), v.reshape(-1)).reshape(ns + 3, ny, nx)


def _band(seed, nx, ny, ns):
    """(NS + 3, ny, nx): unburnt gas at 1 atm / 298 K with a band of one column in 32 at 40
    atm / 3000 K whose density varies by 1% from cell to cell."""
    g = _gen(seed)
    hot = (torch.arange(nx, device="cuda") < max(4, nx // 32))[None, :].expand(ny, nx).reshape(-1)
    one = torch.ones(nx * ny, dtype=torch.float64, device="cuda")
    U = _conserved(torch.where(hot, 3000.0 * one, 298.0 * one), torch.where(hot, 40.0 * ATM * one, ATM * one),
                   _mole(FRESH, ns)[:, None] * one, 0 * one, 0 * one)
    return (U * torch.where(hot, _uniform(g, nx * ny, 0.99, 1.01), one)).reshape(ns + 3, ny, nx)


def _cells(case, seed):
    """(NS + 3, n) states and the intervals (per cell or one) of a batch."""
    g, n, ns = _gen(seed), case["cells"], case["ns"]
    field = case.get("field", "front")
    if field == "front":
        # a level of about 4 : 1 cut to n cells (row by row, so a last row may be short)
        ny = max(1, int(round(math.sqrt(n / 4.0))))
        nx = -(-n // ny)
        return _front(seed, nx, ny, ns, 1e-4).reshape(ns + 3, -1)[:, :n].contiguous(), 2.5e-8
    z = torch.zeros(n, dtype=torch.float64, device="cuda")
    X = torch.zeros(ns, n, dtype=torch.float64, device="cuda")
    if field == "uneven":
        T, p = _uniform(g, n, 800.0, 2500.0), ATM * _log_uniform(g, n, 0.1, 10.0)
        phi, dil = _log_uniform(g, n, 0.3, 3.0), _uniform(g, n, 0.0, 0.8)
        X[0], X[1] = (1 - dil) * 2 * phi / (2 * phi + 1), (1 - dil) / (2 * phi + 1)
        X[ns - 1] += dil
        return _conserved(T, p, X, z, z), _log_uniform(g, n, 1e-7, 1e-6)
    T, p, phi = _uniform(g, n, 1000.0, 1500.0), ATM * _uniform(g, n, 1.0, 5.0), _uniform(g, n, 0.5, 2.0)
    X[0], X[1], X[8] = 2 * phi, 1.0, 3.76
    if field == "kernel":  # an ignition kernel: radicals present
        X[3], X[4], X[5] = 0.05, 0.03, 0.05
    return _conserved(T, p, X / X.sum(0), z, z), 5e-7


def _wedge(nx, ny):
    """Level keys and free stream of the Mach 7 flow over a 30 degree wedge (9 species)."""
    from hyperflow_gb300 import workloads as W
    U, lv = W.wedge(nx=nx, ny=ny)
    return U, lv


def _flow_inputs(case, seed):
    """(U (NV, ny, nx), level keys) of a flow case."""
    nx, ny, ns = case["nx"], case["ny"], case["ns"]
    if not case["wedge"]:
        U = _front(seed, nx, ny, ns, 1e-4)
        inlet = [float(t) for t in U[:, 0, nx - 1].cpu()]
        return U, dict(nx=nx, ny=ny, dx=1e-4, dy=1e-4, periodic=(0, 1), boundary_lo=("reflecting", "reflecting"),
                       boundary_hi=("transmissive", "reflecting"), inlet=inlet)
    g = _gen(seed)
    dx = 0.032 / 512
    x = (torch.arange(nx, dtype=torch.float64, device="cuda")[None, :] + 0.5) * dx - 0.004
    y = (torch.arange(ny, dtype=torch.float64, device="cuda")[:, None] + 0.5) * dx
    s = 0.2 * x - y  # > 0: between the wedge surface (the bottom row) and the oblique shock
    behind = s > 0
    prog = torch.where(behind, torch.clamp((x + 0 * y - 0.008) / 0.01, 0.0, 1.0), torch.zeros_like(s))
    noise = 1.0 + 0.02 * (torch.rand(ny, nx, dtype=torch.float64, device="cuda", generator=g) - 0.5)
    T = torch.where(behind, 1300.0 + 1300.0 * prog, torch.full_like(s, 300.0)) * noise
    p = torch.where(behind, 1.6 + 0.4 * prog, torch.full_like(s, 0.1)) * ATM
    V, th = 2850.0, math.radians(30.0)
    u = torch.where(behind, torch.full_like(s, 2100.0), torch.full_like(s, V * math.cos(th)))
    v = torch.where(behind, -120.0 * torch.clamp(y / (0.2 * torch.clamp(x, min=dx)), 0.0, 1.0),
                    torch.full_like(s, -V * math.sin(th)))
    fresh, burnt = (_mole({k: w for k, w in m.items()}, ns) for m in (FRESH, BURNT))
    X = fresh[:, None] * (1 - prog.reshape(-1)) + burnt[:, None] * prog.reshape(-1)
    U = _conserved(T.reshape(-1), p.reshape(-1), X, u.reshape(-1), v.reshape(-1)).reshape(ns + 3, ny, nx)
    one = torch.ones(1, dtype=torch.float64, device="cuda")
    q = _conserved(300.0 * one, 0.1 * ATM * one, fresh[:, None], V * math.cos(th) * one, -V * math.sin(th) * one)[:, 0]
    return U, dict(nx=nx, ny=ny, dx=dx, dy=dx, xlo=-0.004, ylo=0.0, periodic=(0, 0), boundary_lo=("inflow", "wedge"),
                   boundary_hi=("transmissive", "inflow"), inlet=[float(t) for t in q.cpu()], wedge_start=0.0)


def _line(seed, nx, ny):
    """(13, ny, nx): the planar detonation of the front with a resolution-independent shape."""
    return _front(seed, nx, ny, 10, 0.1 / nx)


DET1D = dict(periodic=(0, 0), boundary_lo=("reflecting", "reflecting"), boundary_hi=("transmissive", "reflecting"))


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    import hyperflow_gb300 as hf
    kind = case["kind"]
    ns = case.get("ns", {"ignition": 9, "amr": 9, "adjoint": 10}.get(kind, 9))
    ctx = hf.Context("H2_Li" if ns == 9 else "H2_Li+AR")
    s = dict(case=case, hf=hf, ctx=ctx, ns=ns)
    if kind == "eos":
        s["q"] = _cells(dict(case), seed)[0]
    elif kind == "flow":
        U, lv = _flow_inputs(case, seed)
        s["level"] = hf.make_level(**lv)
        a = hf.PatchArray(ns + 3, case["nx"], case["ny"])
        a.interior().copy_(U)
        s["u"] = [a, a.like(), a.like()]
        s["form"] = hf._lib.HF_FLUX_FUSED if case["form"] == "fused" else hf._lib.HF_FLUX_PLAIN
    elif kind == "chem":
        s["U0"], s["dt"] = _cells(case, seed)
        s["U"] = s["U0"].clone()
        s["chem"] = hf.ChemistryBatch(ctx, form=case["form"])
    elif kind == "ignition":
        s["U0"] = _cells(dict(case, ns=9, field="kernel"), seed)[0]
        s["sens"] = hf.ChemSensitivity(ctx, 1e-7, case["ncalls"], objective=case["objective"], ignition_dT=10.0,
                                       checkpoint_every=50)
    elif kind == "strang":
        nx, ny = case["nx"], case["ny"]
        dx = 1e-4 if ny > 2 else 0.1 / nx
        U = _band(seed, nx, ny, ns) if ny > 2 else _front(seed, nx, ny, ns, dx)
        lv = hf.make_level(nx=nx, ny=ny, dx=dx, dy=dx, inlet=[float(t) for t in U[:, 0, nx - 1].cpu()],
                           **(DET1D if ny <= 2 else dict(DET1D, periodic=(0, 1))))
        s["host"] = U.cpu().pin_memory()
        s["step"] = hf.Stepper(ctx, lv, U, flux="plain", chem="batched")
    elif kind == "amr":
        U, lv = _wedge(case["nx"], case["ny"])
        g = np.random.default_rng(seed)
        U = U * (1.0 + 0.01 * g.uniform(-1.0, 1.0, size=U.shape[1:]))[None]
        s["amr"] = hf.AmrStepper(ctx, hf.make_level(**lv), torch.from_numpy(U).cuda(), max_level=2, block=32,
                                 tag_buffer=2, regrid_interval=case["steps"],
                                 tags=dict(pressure_tag=0.5, temperature_tag=0.5, fuel_rate_tag=1e30, density_tag=0.05,
                                           box=(-0.001, 0.002, 0.0, 0.002)))
    else:
        U = _line(seed, case["nx"], case["ny"])
        s["dx"] = 0.1 / case["nx"]
        s["level"] = hf.make_level(nx=case["nx"], ny=case["ny"], dx=s["dx"], dy=s["dx"],
                                   inlet=[float(t) for t in U[:, 0, -1].cpu()], **DET1D)
        s["U0"] = U
        s["seed"] = torch.randn(U.shape, dtype=torch.float64, device="cuda", generator=_gen(seed + 1)) / U.abs().amax(
            dim=(1, 2), keepdim=True).clamp(min=1e-3)
    return s


def _split(U, ns):
    """A state by its physical parts, each of its own scale."""
    return {"rhoY": U[:ns], "momentum": U[ns:ns + 2], "energy": U[ns + 2]}


def run(s):
    case, hf, ctx, ns = s["case"], s["hf"], s["ctx"], s["ns"]
    kind = case["kind"]
    if kind == "eos":
        p, a, T, status = hf.properties(ctx, s["q"])
        return {"p": p, "a": a, "T": T, "status": status}
    if kind == "flow":
        u, t, o = s["u"]
        h = 0.5 * hf.cfl_dt(ctx, s["level"], u, 0.5)
        plain = case["form"] == "plain"  # the fused kernel resolves the boundaries itself
        if plain:
            hf.fill(ctx, s["level"], u)
        hf.euler_stage(ctx, s["level"], u, t, h, form=s["form"])
        if plain:
            hf.fill(ctx, s["level"], t)
        hf.euler_stage(ctx, s["level"], t, o, h, u_old=u, form=s["form"])
        return {"h": h, "stage": _split(t.interior(), ns), "out": _split(o.interior(), ns)}
    if kind == "chem":
        s["U"].copy_(s["U0"])
        dt = s["dt"]
        if isinstance(dt, float):
            s["chem"].advance(s["U"], dt)
        else:
            s["chem"].advance(s["U"], 0.0, dt_cell=dt)
        return _split(s["U"], ns)
    if kind == "ignition":
        J, G, G0 = s["sens"].adjoint(s["U0"], initial=True)
        return {"J": J, "dJ_dlnA": G, "dJ_dY0": G0}
    if kind == "strang":
        s["step"].set_host(s["host"])
        done = s["step"].run(case["steps"])
        return dict(_split(s["step"].state(), ns), steps=done)
    if kind == "amr":
        dts = [s["amr"].step() for _ in range(case["steps"])]
        out = {"dt": np.array(dts)}
        for lev in range(3):
            U, active = s["amr"].level(lev)
            out["level%d" % lev] = dict(_split(U, ns), active=active)
        return out
    fa = hf.FlowAdjoint(ctx, s["level"], s["U0"], case["steps"], checkpoint_every=2, chemistry=case["chemistry"])
    bar, grad = fa.adjoint(s["seed"])
    out = {"final": _split(fa.final, ns), "U0_bar": bar, "dJ_dlnA": grad, "dts": fa.dts.copy()}
    fa.close()
    return out


# ------------------------------------------------------------------ work
# Double-precision operations that cannot be done without, by count of the formulas: an EOS
# solve (mixture polynomial, two Newton updates, p and a) about 220; a face (reconstruction of
# NV components, two EOS solves, HLLC) 2 x 220 + 16 NV + 60; a cell update about 8 NV; a Rodas4
# step (6 right-hand sides, a Jacobian, an 8 x 8 LU and 6 solves) about 9000; its reverse
# about 5 times that.  The steps a cell takes are the inputs' own: mean counts of the fields.
STEP = 9000.0
STEPS = {"uneven": 60.0, "front": 8.0, "ignition": 12.0}


def work(case):
    kind = case["kind"]
    nv = case.get("ns", 9) + 3
    if kind == "eos":
        n = case["cells"]
        return {"bytes": n * (8.0 * nv + 28.0), "flops": 250.0 * n}
    if kind == "flow":
        n = case["nx"] * case["ny"]
        return {"bytes": 8.0 * nv * n * 6, "flops": n * (2 * (2 * (500.0 + 16 * nv) + 8 * nv) + 250.0)}
    if kind == "chem":
        n = case["cells"]
        return {"bytes": 16.0 * nv * n, "flops": n * STEP * STEPS[case["field"]]}
    if kind == "ignition":
        n = case["cells"]
        return {"bytes": 8.0 * n * (12 + 21 + 9), "flops": n * case["ncalls"] * 12.0 * STEP * 7}
    if kind == "strang":
        n = case["nx"] * case["ny"] * case["steps"]
        return {"bytes": 8.0 * nv * n * 14, "flops": n * (4 * (2 * (500.0 + 16 * nv) + 8 * nv) + STEP * STEPS["front"])}
    if kind == "amr":
        n = case["nx"] * case["ny"] * case["steps"] * 2  # about half the base area holds finer cells
        return {"bytes": 8.0 * 12 * n * 14, "flops": n * (4 * (2 * (500.0 + 16 * 12) + 8 * 12) + 3000.0)}
    n = case["nx"] * case["ny"] * case["steps"]
    return {"bytes": 8.0 * 13 * n * 30, "flops": n * (12 * (2 * 700.0) + (STEP * 8 * 7 if case["chemistry"] else 0.0))}


# ------------------------------------------------------------------ exact values
def _eos(U, ns, T=None):
    """(p, a, T) of states (NS + 3, n): Newton on e(T) to the last bit."""
    W = _species(ns, U.device)[0][:, None]
    rho = U[:ns].sum(0)
    z = U[:ns] / rho / W
    u, v = U[ns] / rho, U[ns + 1] / rho
    e = (U[ns + 2] / rho - 0.5 * (u * u + v * v)) / RU
    T = _newton(z, e, ns, T)
    zs = z.sum(0)
    cv = (z * (_cp_R(T, ns) - 1.0)).sum(0)
    return rho * RU * T * zs, torch.sqrt((cv + zs) / cv * RU * T * zs), T


def _newton(z, e, ns, T=None):
    with torch.no_grad():
        T = torch.full_like(e, 1000.0) if T is None else T
        for _ in range(40):
            f = e - T * (z * (_h_RT(T, ns) - 1.0)).sum(0)
            d = (f / (z * (_cp_R(T, ns) - 1.0)).sum(0)).clamp(-1000.0, 1000.0)
            Tn = torch.where(T + d > 0, T + d, 0.5 * T)
            done = bool(((Tn - T).abs() <= 1e-13 * Tn).all())
            T = Tn
            if done:
                break
    return T


def _minmod(a, b):
    return torch.where(a * b > 0, torch.copysign(torch.minimum(a.abs(), b.abs()), a), torch.zeros_like(a))


def _hllc(l, r, pl, pr, N, ns):
    E = ns + 2
    rl, rr = l[:ns].sum(0), r[:ns].sum(0)
    ul, ur = l[N] / rl, r[N] / rr
    sl = torch.minimum(ul - pl[1], ur - pr[1])
    sr = torch.maximum(ul + pl[1], ur + pr[1])

    def physical(q, v, p):
        f = v * q
        f[N] += p
        f[E] += p * v
        return f

    fl, fr = physical(l, ul, pl[0]), physical(r, ur, pr[0])
    dl, dr = rl * (sl - ul), rr * (sr - ur)
    sm = (pr[0] - pl[0] + dl * ul - dr * ur) / (dl - dr)

    def star(q, f, v, s, p, rho):
        scale = (s - v) / (s - sm)
        st = q * scale
        rs = rho * scale
        st[N] = rs * sm
        st[E] = q[E] * scale + rs * (sm - v) * (sm + p / (rho * (s - v)))
        return f + s * (st - q)

    mid = torch.where(sm >= 0, star(l, fl, ul, sl, pl[0], rl), star(r, fr, ur, sr, pr[0], rr))
    return torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, mid))


def _ghosted(U, lv, ns):
    """U (NV, ny, nx) with two ghost layers (corner cells unused) by the level's boundary keys."""
    nv, ny, nx = U.shape
    G = torch.zeros(nv, ny + 4, nx + 4, dtype=U.dtype, device=U.device)
    G[:, 2:-2, 2:-2] = U
    inlet = torch.tensor(lv["inlet"], dtype=U.dtype, device=U.device)[:, None]
    for d in range(2):
        n = nx if d == 0 else ny
        A = G[:, 2:-2, :] if d == 0 else G[:, :, 2:-2].transpose(1, 2)
        src = A.clone()
        for hi in range(2):
            kind = (lv["boundary_hi"] if hi else lv["boundary_lo"])[d]
            for k in range(2):
                at = 2 + n + k if hi else 1 - k
                edge, image = (1 + n, 1 + n - k) if hi else (2, 2 + k)
                if lv["periodic"][d]:
                    A[:, :, at] = src[:, :, 2 + (k % n) if hi else 1 + n - (k % n)]
                elif kind == "inflow":
                    A[:, :, at] = inlet
                elif kind == "transmissive":
                    A[:, :, at] = src[:, :, edge]
                else:
                    m = src[:, :, image].clone()
                    m[ns + d] = -m[ns + d]
                    if kind == "wedge":
                        x = lv["xlo"] + (torch.arange(nx, dtype=U.dtype, device=U.device) + 0.5) * lv["dx"]
                        m = torch.where((x >= lv["wedge_start"])[None], m, src[:, :, edge])
                    A[:, :, at] = m
    return G


def _stage(U, lv, ns, h):
    """One Euler stage of (NV, ny, nx)."""
    G = _ghosted(U, lv, ns)
    nv, ny, nx = U.shape
    out = U.clone()
    for d in range(2):
        A = G[:, 2:-2, :] if d == 0 else G[:, :, 2:-2].transpose(1, 2)  # (NV, rows, n + 4)
        n = nx if d == 0 else ny
        qa, qb, qc, qd = (A[:, :, k:k + n + 1] for k in range(4))
        l = qb + 0.5 * _minmod(qb - qa, qc - qb)
        r = qc - 0.5 * _minmod(qc - qb, qd - qc)
        shape = l.shape
        l, r = l.reshape(nv, -1), r.reshape(nv, -1)
        pl, pr = _eos(l, ns), _eos(r, ns)
        f = _hllc(l, r, pl, pr, ns + d, ns).reshape(shape).clone()
        x = lv.get("xlo", 0.0) + (torch.arange(nx, dtype=U.dtype, device=U.device) + 0.5) * lv["dx"]
        for hi, at in ((0, 0), (1, n)):
            kind = (lv["boundary_hi"] if hi else lv["boundary_lo"])[d]
            if lv["periodic"][d] or kind not in ("reflecting", "wedge"):
                continue
            keep = torch.zeros(nv, 1, dtype=U.dtype, device=U.device)
            keep[ns + d] = 1.0
            wall = f[:, :, at] * keep
            f[:, :, at] = torch.where((x >= lv["wedge_start"])[None], wall, f[:, :, at]) if kind == "wedge" else wall
        df = (f[:, :, 1:] - f[:, :, :-1]) * (h / lv["dx" if d == 0 else "dy"])
        out = out - (df if d == 0 else df.transpose(1, 2))
    return out


def _cfl(U, lv, ns, cfl):
    Uf = U.reshape(ns + 3, -1)
    _, a, _ = _eos(Uf, ns)
    rho = Uf[:ns].sum(0)
    rate = ((Uf[ns] / rho).abs() + a) / lv["dx"] + ((Uf[ns + 1] / rho).abs() + a) / lv["dy"]
    return cfl / float(rate.max())


def _reactions(ns, device):
    """Stoichiometry and rate data as arrays: the mechanism file's 21 reactions."""
    R = []
    for r in _fixture()["reactions"]:
        eq = r["equation"].replace("(+ M)", "").replace(" + M", "")
        sides = [[n.strip() for n in part.split("+") if n.strip()] for part in eq.split("<=>")]
        nu = [[0.0] * ns for _ in range(2)]
        for k, names in enumerate(sides):
            for n in names:
                m = 1.0
                if " " in n:
                    m, n = n.split()
                nu[k][NAMES.index(n)] += float(m)
        eff = [1.0] * ns
        for n, v in (r.get("efficiencies") or {}).items():
            if n in NAMES[:ns]:
                eff[NAMES.index(n)] = v
        k = r.get("rate-constant") or r["high-P-rate-constant"]
        R.append((nu[0], nu[1], eff, k, r.get("low-P-rate-constant"), (r.get("Troe") or {}).get("A"), r["type"]))
    return R


def _rhs(C, rho, e, ns, T, tab):
    """dC/dt (ns, n) at concentrations C, energy e; T: guess in, solution out."""
    W = _species(ns, C.device)[0][:, None]
    z = C / rho
    T = _newton(z, e / RU, ns, T)
    _, lo, hi = _species(ns, C.device)
    a = torch.where((T <= 1000.0)[None, :, None], lo[:, None, :], hi[:, None, :])
    s = (a[..., 0] * torch.log(T) + T * (a[..., 1] + T * (a[..., 2] / 2 + T * (a[..., 3] / 3 + T * a[..., 4] / 4)))
         + a[..., 6])
    g = _h_RT(T, ns) - s
    w = torch.zeros_like(C)
    lnT, cal = torch.log(T), 4184.0 / RU
    arr = lambda k: k["A"] * torch.exp(k["b"] * lnT - k["Ea"] * cal / T)  # noqa: E731
    for f, b, eff, k, k0, troe, kind in tab:
        kf = arr(k)
        if k0 is not None or "three" in kind:
            M = (C * torch.tensor(eff, dtype=C.dtype, device=C.device)[:, None]).sum(0)
        if k0 is not None:
            Pr = arr(k0) * M / kf
            lF = math.log10(troe)
            c, nn = -0.4 - 0.67 * lF, 0.75 - 1.27 * lF
            x = torch.log10(Pr.clamp(min=1e-300)) + c
            kf = kf * Pr / (1 + Pr) * 10.0 ** (lF / (1 + (x / (nn - 0.14 * x)) ** 2))
        elif "three" in kind:
            kf = kf * M
        dn = sum(b) - sum(f)
        lnK = sum((fi - bi) * g[i] for i, (fi, bi) in enumerate(zip(f, b)) if fi != bi) + dn * torch.log(ATM / (RU * T))
        q = torch.ones_like(T)
        p = torch.exp(-lnK)
        for i, (fi, bi) in enumerate(zip(f, b)):
            for _ in range(int(fi)):
                q = q * C[i]
            for _ in range(int(bi)):
                p = p * C[i]
        q = kf * (q - p)
        for i, (fi, bi) in enumerate(zip(f, b)):
            if fi != bi:
                w[i] += (bi - fi) * q
    return w, T


def _react(U, ns, dt, steps):
    """Linearly implicit Euler with extrapolation (harmonic sequence to order 8) over `steps`
    equal intervals of dt: concentrations at constant density and energy."""
    W = _species(ns, U.device)[0][:, None]
    rho = U[:ns].sum(0)
    e = U[ns + 2] / rho - 0.5 * ((U[ns] / rho) ** 2 + (U[ns + 1] / rho) ** 2)
    C = U[:ns] / W
    tab = _reactions(ns, U.device)
    T = None
    n = C.shape[1]
    eye = torch.eye(ns, dtype=C.dtype, device=C.device)
    H = dt / steps
    for _ in range(steps):
        f0, T = _rhs(C, rho, e, ns, T, tab)
        d = 1e-7 * C.clamp(min=1e-9 * float(C.max()))
        many = torch.cat([C + eye[:, k:k + 1] * d[k] for k in range(ns)], 1)
        f1, _ = _rhs(many, rho.repeat(ns), e.repeat(ns), ns, T.repeat(ns), tab)
        J = ((f1.reshape(ns, ns, n) - f0[:, None]) / d[None]).permute(2, 0, 1)
        table = []
        for k in range(1, 9):
            hk = H / k
            lu = torch.linalg.lu_factor(eye - hk * J)
            y, f = C, f0
            for i in range(k):
                if i:
                    f, _ = _rhs(y, rho, e, ns, T, tab)
                y = y + torch.linalg.lu_solve(*lu, (hk * f).T[..., None])[..., 0].T
            row = [y]
            for j in range(1, k):
                row.append(row[j - 1] + (row[j - 1] - table[-1][j - 1]) / (k / (k - j) - 1.0))
            table.append(row)
        C = table[-1][-1]
    out = U.clone()
    out[:ns] = C * W
    return out


def exact(case, seed):
    kind = case["kind"]
    ns = case.get("ns", 9)
    if kind == "eos":
        q = _cells(dict(case), seed)[0]
        p, a, T = _eos(q, ns)
        return {"p": p, "a": a, "T": T, "status": torch.zeros(q.shape[1], dtype=torch.int32, device="cuda")}
    if kind == "flow":
        U, lv = _flow_inputs(case, seed)
        h = 0.5 * _cfl(U, lv, ns, 0.5)
        t = _stage(U, lv, ns, h)
        o = 0.5 * U + 0.5 * _stage(t, lv, ns, h)
        return {"h": h, "stage": _split(t, ns), "out": _split(o, ns)}
    if kind == "chem" and case["field"] == "ignition" and case["cells"] <= 20000:
        # intervals halved until two resolutions agree
        U, dt = _cells(case, seed)
        last, m = _react(U, ns, dt, 8), 16
        while m <= 64:
            now = _react(U, ns, dt, m)
            if float(((now - last).abs().amax(1) / now.abs().amax(1).clamp(min=1e-300)).max()) < 1e-10:
                return _split(now, ns)
            last, m = now, 2 * m
        return None
    # adaptive runs of many steps, their reverse sweeps and hierarchies: no value in 20 seconds
    return None
