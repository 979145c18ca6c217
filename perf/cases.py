"""The measured work of this framework: what its users have it do, through its public entry points.

Three kinds of program use it: drivers of the SPH impact solver (one impact, a batch, a served request, a
host that owns the state), drivers of the Eulerian grid solver (3-D impacts, axisymmetric craters, gas
tests), and code that uses the device cell sort alone.  Sizes come from the workloads of `deorbit_gb300.ic`
and `deorbit_gb300.grid_ic`, the tests and the benchmark.

A case is a dict: "kind" plus the sizes and options of that kind.
  sph_run    one impact in a Context: `steps` steps per pass, driven by the device's CFL step (run) or by the
             host (timestep / step); "rewind" writes the stored start back first (a sweep over one start).
  sph_batch  `count` impacts of uneven sizes in one Context, `steps` steps per pass.
  sph_host   step_fields: the state comes from host arrays and goes back to them in every step.
  sph_serve  a resident server: `count` requests submitted, run for `steps` steps each and collected.
  grid       the grid solver: `steps` steps of the drivers' loop per pass, then the fields are read.
  sort       cell_sort on device arrays.

The mixed forms compute pair sums and fluxes in FP32, so a program takes their results as FP32; the FP64
forms' results are FP64.  Damage is on in the FP64 cases and in the mixed cases of many particles; the
small mixed ones run hydro or strength alone, because the damage law counts activated flaws, a step
function of the stress: one particle whose FP32 stress lies on a threshold changes a small result by far
more than any rounding does, and nothing could be compared.
"""
import ctypes
import math

import numpy as np
import torch

from deorbit_gb300 import euler, grid_ic, ic, serve, sph

SPH_OUT = ["x", "y", "z", "vx", "vy", "vz", "u", "rho", "hh", "P"]
SPH_OUT_S = ["Sxx", "Syy", "Szz", "Sxy", "Sxz", "Syz"]
SPH_STATE = ["x", "y", "z", "vx", "vy", "vz", "u", "hh", "ax", "ay", "az", "dudt"]
SPH_STATE_S = SPH_OUT_S + ["dSxx", "dSyy", "dSzz", "dSxy", "dSxz", "dSyz"]
BATCH_OUT = ["x", "y", "z", "vx", "vy", "vz", "u", "rho", "D"]
GRID_OUT = ["r", "mu", "mv", "mw", "E", "Sxx", "Syy", "Szz", "Sxy", "Sxz", "Syz", "D", "rc"]
GRID_OUT_AF = GRID_OUT + ["af", "vib"]


def listed():
    return [
        # the plain FP64 solver on the hydro-only half-space impact, 48 x 48 x 24 target, stepped by its host
        dict(name="sph_fp64_halfspace_57k", kind="sph_run", ic="halfspace", form="fp64", n=57472, strength=False,
             damage=False, drive="host", rewind=False, steps=2),
        # FP64 grazing impact with strength and multi-flaw damage (the checked form of the large workload)
        dict(name="sph_fp64_grazing_131k", kind="sph_run", ic="grazing", form="fp64", n=131072, strength=True,
             damage=True, drive="device", rewind=False, steps=2),
        # the benchmark's workload: 1,048,576 particles, strength + damage, mixed form
        dict(name="sph_mixed_grazing_1m", kind="sph_run", ic="grazing", form="mixed", n=1 << 20, strength=True,
             damage=True, drive="device", rewind=False, steps=8),
        # a sweep of small impacts from one stored start: the smallest runs, where launches and latency count
        dict(name="sph_mixed_small_6k", kind="sph_run", ic="impact", form="mixed", n=6000, strength=True,
             damage=False, drive="device", rewind=True, steps=16),
        # batched sweep: impacts of 5k-80k particles in one launch sequence
        dict(name="sph_mixed_batch_24", kind="sph_batch", form="mixed", count=24, lo=5000, hi=80000, steps=8),
        # a host program that owns the state: fields up, one step, fields down
        dict(name="sph_mixed_host_step_262k", kind="sph_host", ic="grazing", form="mixed", n=262144, strength=True,
             damage=False),
        # served requests, whole life: submit, admit, initialise, 20 steps, results on the host
        dict(name="sph_serve_20k", kind="sph_serve", form="mixed", count=2, n=20000, strength=True, steps=20),
        # 3-D half-space impact on the grid solver, ROCK yield + damage + gravity, reference arithmetic
        dict(name="grid_fp64_impact_96", kind="grid", problem="impact3d", form="fp64", N=96, steps=1),
        # the same in the mixed form on a larger grid
        dict(name="grid_mixed_impact_160", kind="grid", problem="impact3d", form="mixed", N=160, steps=8),
        # the crater driver's default size (150 x 110, axisymmetric) with explicit fluidization
        dict(name="grid_fp64_crater_150x110", kind="grid", problem="crater", form="fp64", cppr=10, visc=False,
             steps=10),
        # a quick-look crater (60 x 44) with the implicit viscosity: the smallest grids
        dict(name="grid_mixed_crater_60x44", kind="grid", problem="crater", form="mixed", cppr=4, visc=True,
             steps=10),
        # the radix cell sort as a primitive, odd size, about two particles per cell
        dict(name="cell_sort_3m", kind="sort", n=3000017, per_cell=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sph_run", "sph_run", "sph_run", "sph_batch", "sph_host", "sph_serve", "grid", "grid", "grid",
                       "grid", "sort"])
    if kind == "sph_run":
        form = rng.choice(["fp64", "mixed"])
        if form == "fp64":
            n = _log_int(rng, 1500, 130000)
            which = rng.choice(["halfspace", "grazing", "impact"]) if n > 20000 else "impact"
            strength = which != "halfspace" and rng.random() < 0.7
            return dict(kind=kind, ic=which, form=form, n=n, strength=strength,
                        damage=strength and rng.random() < 0.7, drive=rng.choice(["host", "device"]),
                        rewind=n < 20000, steps=rng.randint(1, 4))
        n = _log_int(rng, 1500, 1000000)
        which = "grazing" if n > 200000 else rng.choice(["impact", "halfspace"])
        strength = which == "grazing" or (which == "impact" and rng.random() < 0.5)
        return dict(kind=kind, ic=which, form=form, n=n, strength=strength, damage=n > 200000,
                    drive=rng.choice(["host", "device"]), rewind=n < 200000, steps=rng.randint(4, 16))
    if kind == "sph_batch":
        lo = _log_int(rng, 5000, 20000)
        return dict(kind=kind, form="mixed", count=rng.randint(16, 24), lo=lo, hi=4 * lo, steps=rng.randint(2, 8))
    if kind == "sph_host":
        return dict(kind=kind, ic="impact", form=rng.choice(["fp64", "mixed", "mixed"]), n=_log_int(rng, 3000, 120000),
                    strength=rng.random() < 0.5, damage=False)
    if kind == "sph_serve":
        return dict(kind=kind, form="mixed", count=rng.randint(1, 4), n=_log_int(rng, 5000, 60000),
                    strength=rng.random() < 0.5, steps=rng.randint(8, 24))
    if kind == "grid":
        problem = rng.choice(["impact3d", "impact3d", "crater", "crater", "sedov", "sod"])
        form = rng.choice(["fp64", "mixed"])
        if problem == "impact3d":
            return dict(kind=kind, problem=problem, form=form, N=_log_int(rng, 24, 96 if form == "fp64" else 160),
                        steps=rng.randint(1, 2) if form == "fp64" else rng.randint(2, 8))
        if problem == "crater":
            return dict(kind=kind, problem=problem, form=form, cppr=rng.randint(3, 14), visc=rng.random() < 0.4,
                        steps=rng.randint(4, 16))
        if problem == "sedov":
            return dict(kind=kind, problem=problem, form=form, N=_log_int(rng, 16, 96), steps=rng.randint(1, 4))
        return dict(kind=kind, problem=problem, form=form, N=_log_int(rng, 50, 4000), steps=rng.randint(8, 32))
    return dict(kind="sort", n=_log_int(rng, 1000, 6000000), per_cell=rng.choice([1, 2, 4, 8]))


# ---------------------------------------------------------------- inputs

def _scenario(case, seed, n=None):
    """One impact of the case: geometry, angle, speed and lattice jitter from the seed."""
    rng = np.random.default_rng([seed, 17])
    n = n or case["n"]
    strength = bool(case.get("strength"))
    if case.get("ic") == "halfspace":
        nz = max(6, round((n / 4.15) ** (1 / 3)))  # 48 x 48 x 24 and r = 8 of 57,472, scaled
        sc = ic.impact_halfspace(2 * nz, 2 * nz, nz, r_cells=nz / 3.0, angle_deg=float(rng.uniform(20, 70)),
                                 speed=float(rng.uniform(6000, 10000)), seed=seed)
    elif case.get("ic") == "grazing":
        sc = ic.grazing(n, angle_deg=float(rng.uniform(2, 6)), speed=float(rng.uniform(7000, 9000)), seed=seed)
    else:
        sc = ic.sized_impact(n, seed=seed, angle_deg=float(rng.uniform(1, 45)), speed=float(rng.uniform(4000, 12000)),
                             ratio=case.get("ratio", 0.2), strength=strength)
    if not case.get("damage", False):
        sc.params.update(damage_on=0, flaw_model=0)
        sc.flaws = None
    if not strength:
        sc.materials = [ic.granite(strength=False), ic.iron(strength=False)]
    return sc


def _pinned(n, names):
    return {k: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() for k in names}


def _form(case):
    return sph.FP64 if case["form"] == "fp64" else sph.MIXED


def _taken(case, outs):
    """Host fields as the program keeps them: FP32 from the mixed form, FP64 from the plain one."""
    if case["form"] == "fp64":
        return outs
    return {k: torch.from_numpy(v).float() for k, v in outs.items()}


def _sph_names(case):
    out = SPH_OUT + (SPH_OUT_S if case["strength"] else []) + (["D"] if case.get("damage") else [])
    state = SPH_STATE + (SPH_STATE_S if case["strength"] else []) + (["D"] if case.get("damage") else [])
    return out, state


def _grid_case(case, seed):
    rng = np.random.default_rng([seed, 23])
    p = case["problem"]
    if p == "impact3d":
        g = grid_ic.impact3d(case["N"], speed=float(rng.uniform(6000, 12000)), angle_deg=float(rng.uniform(10, 60)))
    elif p == "crater":  # the crater driver's geometry: 15 x 11 radii, fluidization with its defaults
        g = grid_ic.crater(cppr=case["cppr"], Rfac=15, Zfac=11, U=float(rng.uniform(8000, 15000)), tdec=40.0,
                           eta_af=1e9, visc_imp=int(case["visc"]))
        g.pin_floor, g.sponge_from = 2, int(0.85 * g.shape[0])
    elif p == "sedov":
        g = grid_ic.sedov(case["N"])
        g.fields["E"] = g.fields["E"] * rng.uniform(0.5, 2.0)
        g.fields["r"] = g.fields["r"] * (1 + 0.01 * rng.standard_normal(g.n))
    else:
        g = grid_ic.sod(case["N"])
        g.fields["r"] = g.fields["r"] * rng.uniform(0.8, 1.25)
        g.fields["E"] = g.fields["E"] * rng.uniform(0.8, 1.25)
    g.t_end = 1e30  # a pass is a number of steps
    return g


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        cells = max(1, case["n"] // case["per_cell"])
        return dict(case=case, keys=torch.randint(0, cells, (case["n"],), generator=g, device="cuda",
                                                  dtype=torch.int32),
                    cells=cells, perm=torch.empty(case["n"], dtype=torch.int32, device="cuda"),
                    start=torch.empty(cells + 1, dtype=torch.int32, device="cuda"))
    if kind == "grid":
        gc = _grid_case(case, seed)
        g = euler.from_case(gc, form=euler.FP64 if case["form"] == "fp64" else euler.MIXED)
        if gc.pin_floor or gc.sponge_from >= 0:
            g.set_driver(gc.pin_floor, gc.sponge_from, gc.driver_flags)
        names = GRID_OUT_AF if case["problem"] == "crater" else GRID_OUT
        return dict(case=case, grid=g, cfl=gc.cfl, outs=_pinned(gc.n, names))
    if kind == "sph_serve":
        scs = [_scenario(case, seed + 1 + i, int(case["n"] * (0.7, 1.3, 0.9, 1.1)[i % 4]))
               for i in range(case["count"])]
        fields = SPH_OUT + (SPH_OUT_S if case["strength"] else [])
        return dict(case=case, server=serve.Server(_form(case), fields=fields), scenarios=scs)
    ctx = sph.Context(_form(case))
    if kind == "sph_batch":
        rng = np.random.default_rng(case["count"] * 100003 + case["lo"])  # sizes belong to the case
        ids, bs, ns = {}, [], []
        for i in range(case["count"]):
            n = int(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))
            sc = _scenario(dict(strength=True, damage=True, ratio=float(rng.uniform(0.1, 0.3))), seed + 1 + i, n)
            bs.append(ic.to_context(ctx, sc, material_ids=ids))
            ns.append(sc.n)
        ctx.init()
        # one array per field for all impacts, each reading into its own slice
        outs, at = _pinned(sum(ns), BATCH_OUT), np.cumsum([0] + ns)
        return dict(case=case, ctx=ctx, outs=outs,
                    parts=[(b, [outs[k][at[i]:at[i + 1]] for k in BATCH_OUT]) for i, b in enumerate(bs)])
    sc = _scenario(case, seed)
    b = ic.to_context(ctx, sc)
    ctx.init()
    out, state = _sph_names(case)
    st = dict(case=case, ctx=ctx, b=b, outs=_pinned(sc.n, out))
    if kind == "sph_host":
        st["outs"] = _pinned(sc.n, state + ["rho", "P"])
    if kind == "sph_host" or case["rewind"]:
        st["start"] = _pinned(sc.n, state)
        ctx.read_many(b, state, [st["start"][k] for k in state])
        if kind == "sph_run":  # the step of the stored start is found again by its first force pass
            st["dt0"] = ctx.timestep(b)
    return st


# ---------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        sph.check(sph.lib().sph_cell_sort(state["keys"].data_ptr(), case["n"], state["cells"],
                                          state["perm"].data_ptr(), state["start"].data_ptr(),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return dict(perm=state["perm"], start=state["start"])
    if kind == "grid":
        state["grid"].run(state["cfl"], 1e30, case["steps"])
        return _taken(case, state["grid"].read_many(list(state["outs"]), list(state["outs"].values())))
    if kind == "sph_serve":
        srv = state["server"]
        reqs = [srv.submit(sc, case["steps"]) for sc in state["scenarios"]]
        srv.serve()
        return [_taken(case, r.result) for r in reqs]
    ctx = state["ctx"]
    if kind == "sph_batch":
        ctx.run(case["steps"])
        for b, part in state["parts"]:
            ctx.read_many(b, BATCH_OUT, part)
        return _taken(case, state["outs"])
    b, outs = state["b"], state["outs"]
    if kind == "sph_host":
        _, got = ctx.step_fields(b, state["start"], list(outs), list(outs.values()))
        return _taken(case, got)
    left = case["steps"]
    if case["rewind"]:
        ctx.write_many(b, state["start"])
        ctx.step(state["dt0"])
        left -= 1
    if case["drive"] == "device":
        if left:
            ctx.run(left)
    else:
        for _ in range(left):
            ctx.step(ctx.timestep(b))
    return _taken(case, ctx.read_many(b, list(outs), list(outs.values())))


# ---------------------------------------------------------------- bytes and operations a pass needs

PAIRS = 78  # list entries per particle at h = 1.3 dx


def work(case):
    kind = case["kind"]
    if kind == "sort":  # keys in, order and cell starts out
        cells = max(1, case["n"] // case["per_cell"])
        return {"bytes": 8 * case["n"] + 4 * (cells + 1), "flops": 0}
    if kind == "grid":
        cells, cyl = _grid_cells(case), case["problem"] == "crater"
        word = 8
        outs = len(GRID_OUT_AF if cyl else GRID_OUT)
        state = 16 if case["problem"] in ("impact3d", "crater") else 6
        dirs = 3 if case["problem"] in ("impact3d", "sedov") else (2 if cyl else 1)
        flops = 2 * (dirs * 330 + (350 if state == 16 else 40))  # two Lops: faces and right-hand side
        return {"bytes": cells * word * (2 * state * case["steps"] + 2 * outs), "flops": cells * flops * case["steps"]}
    per = (270 if case["form"] == "mixed" else 426) if case.get("strength", True) else (160 if case["form"] == "mixed" else 250)
    flops = PAIRS * (2 * 25 + (169 if case.get("strength", True) else 110))  # two density iterations, one force pass
    if kind == "sph_batch":
        n = case["count"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": n * (per * case["steps"] + 16 * len(BATCH_OUT)), "flops": n * flops * case["steps"]}
    if kind == "sph_serve":
        n = case["n"] * case["count"]
        return {"bytes": n * (per * case["steps"] + 8 * 10 + 16 * 10), "flops": n * flops * (case["steps"] + 1)}
    out, st = _sph_names(case)
    if kind == "sph_host":
        return {"bytes": case["n"] * (per + 16 * (2 * len(st) + 2)), "flops": case["n"] * flops}
    io = 16 * len(out) + (16 * len(st) if case["rewind"] else 0)
    return {"bytes": case["n"] * (per * case["steps"] + io), "flops": case["n"] * flops * case["steps"]}


def _grid_cells(case):
    if case["problem"] == "crater":
        return (15 * case["cppr"]) * (11 * case["cppr"])
    return case["N"] if case["problem"] == "sod" else case["N"] ** 3


# ---------------------------------------------------------------- the same in 64 bits, in plain torch

def exact(case, seed):
    """What run() returns, from plain torch in FP64: the SPH step without damage, and the grid solver without
    the implicit viscosity (whose solves stop at a tolerance)."""
    kind = case["kind"]
    if kind == "sph_run" and not case["damage"] and case["n"] <= 70000:
        sc = _scenario(case, seed)
        return _exact_sph(sc, case["steps"], _sph_names(case)[0])
    if kind == "sph_host" and not case["damage"] and case["n"] <= 70000:
        return _exact_sph(_scenario(case, seed), 1, _sph_names(case)[1] + ["rho", "P"])
    if kind == "grid" and not case.get("visc"):
        gc = _grid_case(case, seed)
        f = _ExactGrid(gc).run(case["steps"])
        names = GRID_OUT_AF if case["problem"] == "crater" else GRID_OUT
        return {k: f[k].reshape(-1).cpu().numpy() for k in names}
    return None


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev())


def _pairs(x, reach):
    """All pairs (i, j), itself included, closer than `reach`, by comparing blocks."""
    gi, gj = [], []
    for s in range(0, x.shape[0], 1024):
        d = sum((x[s:s + 1024, None, a] - x[None, :, a]) ** 2 for a in range(3))
        i, j = torch.nonzero(d < reach * reach, as_tuple=True)
        gi.append(i + s)
        gj.append(j)
    return torch.cat(gi), torch.cat(gj)


def _tillotson(m, rho, u):
    """Pressure and sound speed of the Tillotson material columns m."""
    eta = rho / m["rho0"]
    mu, w = eta - 1, 1 + u / (m["u0"] * eta * eta)
    dw = -2 * u / (m["u0"] * eta ** 3 * m["rho0"])
    aob = m["a"] + m["b"] / w
    Pc = aob * rho * u + m["A"] * mu + m["B"] * mu * mu
    cu = aob * rho - m["b"] * rho * u / (w * w * m["u0"] * eta * eta)
    cr = aob * u - rho * u * m["b"] / (w * w) * dw + m["A"] / m["rho0"] + 2 * m["B"] * mu / m["rho0"]
    z = m["rho0"] / rho - 1
    dz = -m["rho0"] / (rho * rho)
    e1, e2 = torch.exp(-m["alpha"] * z * z), torch.exp(-m["beta"] * z)
    g = m["b"] * rho * u / w + m["A"] * mu * e2
    Pe = m["a"] * rho * u + g * e1
    eu = m["a"] * rho + (m["b"] * rho / w - m["b"] * rho * u / (w * w * m["u0"] * eta * eta)) * e1
    gr = m["b"] * u / w - m["b"] * rho * u / (w * w) * dw + m["A"] * e2 / m["rho0"] - m["A"] * mu * e2 * m["beta"] * dz
    er = m["a"] * u + gr * e1 - g * e1 * 2 * m["alpha"] * z * dz
    f = (m["ucv"] - m["uiv"])
    cold = (rho >= m["rho0"]) | (u <= m["uiv"])
    hot = u >= m["ucv"]

    def pick(c, e, mix):
        return torch.where(cold, c, torch.where(hot, e, mix))

    P = pick(Pc, Pe, ((u - m["uiv"]) * Pe + (m["ucv"] - u) * Pc) / f)
    dr = pick(cr, er, ((u - m["uiv"]) * er + (m["ucv"] - u) * cr) / f)
    du = pick(cu, eu, ((Pe + (u - m["uiv"]) * eu) + (-Pc + (m["ucv"] - u) * cu)) / f)
    return P, torch.sqrt(torch.clamp(dr + P / (rho * rho) * du, min=1e-6))


def _exact_sph(sc, steps, names):
    """The kick-drift-kick step with adaptive h, artificial viscosity, artificial and deviatoric stress."""
    p = sc.params
    x, v = _t(sc.pos), _t(sc.vel)
    lo, hi = _t(sc.lo), _t(sc.hi)
    mass, u = _t(sc.mass), _t(sc.u)
    n = x.shape[0]
    mid = _t(sc.mat, torch.int64)
    m = {k: _t([d[k] for d in sc.materials])[mid] for k in ic.MAT_FIELDS}
    h = torch.full_like(u, p["h_init"])
    h0 = h.clone()
    S, dS = torch.zeros(6, n, device=x.device, dtype=x.dtype), torch.zeros(6, n, device=x.device, dtype=x.dtype)
    q0 = 1 / p["eta"]
    w0 = 1 - 1.5 * q0 * q0 + 0.75 * q0 ** 3
    eps_as = p.get("eps_as", 0.0)
    move = (_t(sc.fixed, torch.int64) == 0)

    def density(x, h):
        for _ in range(4):
            hmax = h.max()
            # the reference looks in the 27 cells around a particle's own, of a width that fits 2 h_max
            ext = hi - lo
            nc = torch.clamp(torch.floor(ext / (2 * hmax)), min=1)
            cell = torch.minimum(torch.clamp(torch.floor((x - lo) / (ext / nc)), min=0), nc - 1)
            i, j = _pairs(x, 3.0 * float(hmax))
            near = ((cell[i] - cell[j]).abs() <= 1).all(dim=1)
            i, j = i[near], j[near]
            r = (x[i] - x[j]).norm(dim=1)
            for _ in range(2):
                own = h[i]
                q = r / own
                t, a = torch.clamp(2 - q, min=0), torch.clamp(1 - q, min=0)
                w = mass[j] / (math.pi * own ** 3) * (0.25 * t ** 3 - a ** 3)
                rho = torch.zeros_like(h).index_add_(0, i, w).clamp(min=1e-30)
                h = torch.minimum(2 * h0, torch.maximum(0.5 * h0, p["eta"] * (mass / rho) ** (1 / 3)))
            if h.max() <= hmax * 1.02:
                break
        return rho, h

    def forces(x, v, u, rho, h, S):
        P, cs = _tillotson(m, rho, u)
        csig = torch.sqrt(cs * cs + (4 / 3) * m["G"] / rho)
        i, j = _pairs(x, 2 * float(h.max()))
        d = x[i] - x[j]
        r = d.norm(dim=1)
        ok = (r < h[i] + h[j]) & (r > 0)
        i, j, d, r = i[ok], j[ok], d[ok], r[ok]
        hb = 0.5 * (h[i] + h[j])
        q = r / hb
        t, a = torch.clamp(2 - q, min=0), torch.clamp(1 - q, min=0)
        dW = (3 * a * a - 0.75 * t * t) / (math.pi * hb ** 4)
        g = d * (dW / r)[:, None]
        dv = v[i] - v[j]
        L = torch.zeros(n, 9, device=x.device, dtype=x.dtype)
        vol = mass / rho
        L.index_add_(0, i, (-(vol[j])[:, None, None] * dv[:, :, None] * g[:, None, :]).reshape(-1, 9))
        L = L.reshape(n, 3, 3)
        dvr = (dv * d).sum(1)
        mu = hb * dvr / (r * r + p["eps"] * hb * hb)
        Pij = torch.where(dvr < 0, (-p["alpha"] * 0.5 * (csig[i] + csig[j]) * mu + p["beta"] * mu * mu) /
                          (0.5 * (rho[i] + rho[j])), torch.zeros_like(mu))
        pr = P / (rho * rho)
        R = torch.where(P < 0, eps_as * -pr, torch.zeros_like(P)) if eps_as > 0 else torch.zeros_like(P)
        term = pr[i] + pr[j] + Pij
        du = torch.zeros_like(u).index_add_(0, i, 0.5 * mass[j] * term * (dv * g).sum(1))
        fr = (0.25 * t ** 3 - a ** 3) / w0
        mt = mass[j] * (term + (R[i] + R[j]) * fr ** 4)
        idx = torch.tensor([[0, 3, 4], [3, 1, 5], [4, 5, 2]], device=x.device)
        T = (S / (rho * rho)).T
        Tij = (T[i] + T[j])[:, idx]
        st = (Tij * g[:, None, :]).sum(2) * mass[j][:, None]
        acc = torch.zeros_like(v).index_add_(0, i, st - g * mt[:, None])
        E, W = 0.5 * (L + L.transpose(1, 2)), 0.5 * (L - L.transpose(1, 2))
        Sm = S.T[:, idx]
        tr = E.diagonal(dim1=1, dim2=2).sum(1) / 3
        J = W @ Sm - Sm @ W
        rate = 2 * m["G"][:, None, None] * (E - tr[:, None, None] * torch.eye(3, device=x.device, dtype=x.dtype)) + J
        solid = m["G"] > 0
        k = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
        dSn = torch.stack([torch.where(solid, rate[:, a_, b_], torch.zeros_like(u)) for a_, b_ in k])
        return P, csig, acc, du + torch.where(solid, (Sm * E).sum((1, 2)) / rho, torch.zeros_like(u)), dSn

    rho, h = density(x, h)
    P, csig, acc, dudt, dS = forces(x, v, u, rho, h, S)
    for _ in range(steps):
        dt = float((p["cfl"] * h / (csig * (1 + p["alpha"]) + 1e-30)).min())
        mv = move[:, None]
        v = torch.where(mv, v + acc * (dt / 2), v)
        x = torch.where(mv, x + v * dt, x)
        rho, h = density(x, h)
        P, csig, acc, dn, dSn = forces(x, v, u, rho, h, S)
        v = torch.where(mv, v + acc * (dt / 2), v)
        u = torch.where(move, torch.clamp(u + 0.5 * dt * (dudt + dn), min=1e-12), u)
        S = torch.where(move, S + 0.5 * dt * (dS + dSn), S)
        Pp = torch.clamp(P, min=0)
        Yc = m["Y0"] + m["mu_i"] * Pp / (1 + m["mu_i"] * Pp / torch.clamp(m["Ylim"] - m["Y0"], min=1.0))
        Y = torch.where(m["yield_model"] == 1, Yc, m["Y"])
        vm = torch.sqrt(3 * (0.5 * (S[:3] ** 2).sum(0) + (S[3:] ** 2).sum(0)))
        S = S * torch.where(Y <= 0, torch.zeros_like(Y), torch.where(vm > Y, Y / vm, torch.ones_like(Y)))
        dudt, dS = dn, dSn
    got = dict(x=x[:, 0], y=x[:, 1], z=x[:, 2], vx=v[:, 0], vy=v[:, 1], vz=v[:, 2], u=u, rho=rho, hh=h, P=P,
               ax=acc[:, 0], ay=acc[:, 1], az=acc[:, 2], dudt=dudt)
    got.update(zip(SPH_OUT_S, S))
    got.update(zip(SPH_STATE_S[6:], dS))
    return {k: got[k].cpu().numpy() for k in names}


class _ExactGrid:
    """The two-stage grid step: limited reconstruction, HLLC and vacuum fluxes, gravity against a hydrostatic
    reference, elastic-plastic strength, tensile damage and shock-activated fluidization."""

    def __init__(self, gc):
        self.c, self.dx = gc, gc.dx
        self.m = {k: float(val) for k, val in gc.material.items()}
        self.p = dict(gz=0.0, tdec=0.0, eta_af=0.0, c_act=0.0, p_coh=1e6, p_act=0.0, rho_cfl=0.0, rho_vac=0.0,
                      y_i0=1e7, mu_i=1.2, mu_d=0.6, y_d0=0.0, y_m=2.5e9, axisym=0, rock=0, af_prel=0, af_seeddp=0)
        self.p.update(gc.params)
        zero = torch.zeros(gc.shape, dtype=torch.float64, device=_dev())
        self.f = {k: zero.clone() for k in euler.FIELDS}
        self.load(gc.fields)
        self.r0 = None
        if gc.set_ref:
            self.r0 = self.f["r"].clone()
            self.p0 = self.pc(self.f)[0]
            self.load(gc.post_ref)
        i = torch.arange(gc.shape[0], dtype=torch.float64, device=_dev())[:, None, None]
        self.i, self.rc = i, (i + 0.5) * self.dx

    def load(self, fields):
        for k, val in fields.items():
            self.f[k] = _t(val).reshape(self.c.shape).clone()

    def eos(self, r, e):
        if self.m["type"] == 0:
            P = (self.m["gamma"] - 1) * r * e
            return torch.clamp(P, min=0), torch.sqrt(torch.clamp(self.m["gamma"] * P / torch.clamp(r, min=1e-30),
                                                                 min=1e-12))
        P, c = _tillotson(self.m, r, e)
        return torch.clamp(P, min=0), c

    def pc(self, s):
        ke = 0.5 * (s["mu"] ** 2 + s["mv"] ** 2 + s["mw"] ** 2) / s["r"]
        return self.eos(s["r"], (s["E"] - ke) / s["r"])

    @staticmethod
    def mm(a, b):
        return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))

    def sides(self, w, ax):
        """Cell values around every face along ax: LL, L, R, RR (the border cell repeated outside)."""
        n = w.shape[ax]
        f = torch.arange(n + 1, device=w.device)
        return [w.index_select(ax, (f + o).clamp(0, n - 1)) for o in (-2, -1, 0, 1)]

    def recon(self, w, ax, floor=None):
        LL, L, R, RR = self.sides(w, ax)
        a, b = L + 0.5 * self.mm(L - LL, R - L), R - 0.5 * self.mm(R - L, RR - R)
        if floor is not None:
            a, b = torch.where(a < floor, L, a), torch.where(b < floor, R, b)
        return a, b

    def vac(self, r, v, t1, t2, e, side):
        p, c = self.eos(r, e)
        g = torch.clamp(torch.clamp(r * c * c / torch.clamp(p, min=1e-30), min=1.01), max=1e5)
        s = side * v
        u0 = 2 / (g + 1) * (c + 0.5 * (g - 1) * s)
        r0 = r * (torch.clamp(u0, min=0) / c) ** (2 / (g - 1))
        p0 = p * (r0 / r) ** g
        out = s - c >= 0
        gone = s + 2 * c / (g - 1) <= 0
        E0 = p0 / (g - 1) + 0.5 * r0 * (u0 * u0 + t1 * t1 + t2 * t2)
        fan = [r0 * side * u0, r0 * u0 * u0 + p0, r0 * side * u0 * t1, r0 * side * u0 * t2, (E0 + p0) * side * u0]
        E = r * e + 0.5 * r * (v * v + t1 * t1 + t2 * t2)
        full = [r * v, r * v * v + p, r * v * t1, r * v * t2, (E + p) * v]
        return [torch.where(out, a, torch.where(gone, torch.zeros_like(b), b)) for a, b in zip(full, fan)]

    def flux(self, A, B, pf=None):
        (rL, vL, aL, bL, eL), (rR, vR, aR, bR, eR) = A, B
        (pL, cL), (pR, cR) = self.eos(rL, eL), self.eos(rR, eR)
        if pf is not None:
            pL, pR = torch.clamp(pf[0], min=0), torch.clamp(pf[1], min=0)
        SL, SR = torch.minimum(vL - cL, vR - cR), torch.maximum(vL + cL, vR + cR)
        Ss = (pR - pL + rL * vL * (SL - vL) - rR * vR * (SR - vR)) / (rL * (SL - vL) - rR * (SR - vR))

        def state(r, v, a, b, e, p):
            E = r * e + 0.5 * r * (v * v + a * a + b * b)
            return [r, r * v, r * a, r * b, E], [r * v, r * v * v + p, r * v * a, r * v * b, (E + p) * v], E

        def star(r, v, a, b, p, S, U, F, E):
            k = r * (S - v) / (S - Ss)
            Us = [k, k * Ss, k * a, k * b, k * (E / r + (Ss - v) * (Ss + p / (r * (S - v))))]
            return [f + S * (us - u_) for f, us, u_ in zip(F, Us, U)]

        UL, FL, EL = state(rL, vL, aL, bL, eL, pL)
        UR, FR, ER = state(rR, vR, aR, bR, eR, pR)
        sL, sR = star(rL, vL, aL, bL, pL, SL, UL, FL, EL), star(rR, vR, aR, bR, pR, SR, UR, FR, ER)
        F = [torch.where(SL >= 0, a, torch.where(SR <= 0, b, torch.where(Ss >= 0, c, d)))
             for a, b, c, d in zip(FL, FR, sL, sR)]
        if pf is None and self.p["rho_vac"] > 0:
            nL, nR = rL < self.p["rho_vac"], rR < self.p["rho_vac"]
            toR, toL = self.vac(*A, 1.0), self.vac(*B, -1.0)
            F = [torch.where(nL & nR, torch.zeros_like(f), torch.where(nR, a, torch.where(nL, b, f)))
                 for f, a, b in zip(F, toR, toL)]
        return F

    def lop(self, s, af):
        p, dx, m = self.p, self.dx, self.m
        r = s["r"]
        V = [s[k] / r for k in ("mu", "mv", "mw")]
        e = (s["E"] - 0.5 * (s["mu"] ** 2 + s["mv"] ** 2 + s["mw"] ** 2) / r) / r
        d = {k: torch.zeros_like(r) for k in euler.RHS}
        mom = ("mu", "mv", "mw")
        for ax in range(3):
            t1, t2 = [(1, 2), (0, 2), (0, 1)][ax]
            q = [self.recon(r, ax, 1e-9), self.recon(V[ax], ax), self.recon(V[t1], ax), self.recon(V[t2], ax),
                 self.recon(e, ax, 0.0)]
            A, B = [a for a, _ in q], [b for _, b in q]
            pf = None
            if ax == 2 and self.r0 is not None:
                dev = self.recon(self.eos(r, e)[0] - self.p0, ax)
                _, cl, cr, _ = self.sides(self.r0, ax)
                pf0 = self.eos(0.5 * (cl + cr), torch.zeros_like(cl))[0]
                pf = (pf0 + dev[0], pf0 + dev[1])
            F = self.flux(A, B, pf)
            _, xl, xr, _ = self.sides(s["rc"] / r, ax)
            F.append(F[0] * torch.where(F[0] >= 0, xl, xr))
            n = r.shape[ax]
            if ax == 0 and p["axisym"]:
                w = torch.arange(n + 1, dtype=r.dtype, device=r.device)[:, None, None] * dx
                D = [-((w * f).narrow(0, 1, n) - (w * f).narrow(0, 0, n)) / (self.rc * dx) for f in F]
                D[1] = D[1] + self.eos(r, e)[0] / self.rc
            else:
                D = [-(f.narrow(ax, 1, n) - f.narrow(ax, 0, n)) / dx for f in F]
            for k, x in zip(("r", mom[ax], mom[t1], mom[t2], "E", "rc"), D):
                d[k] = d[k] + x
        if p["gz"]:
            if self.r0 is None:
                d["mw"] = d["mw"] - p["gz"] * r
            else:
                _, cl, cr, _ = self.sides(self.r0, 2)
                pf0 = self.eos(0.5 * (cl + cr), torch.zeros_like(cl))[0]
                n = r.shape[2]
                d["mw"] = d["mw"] - p["gz"] * (r - self.r0) + (pf0.narrow(2, 1, n) - pf0.narrow(2, 0, n)) / dx
            d["E"] = d["E"] - p["gz"] * s["mw"]
        if m["G"] > 0:
            self.strength(s, af, r, V, d)
        return d

    def strength(self, s, af, r, V, d):
        p, dx, G = self.p, self.dx, self.m["G"]
        void = r < p["rho_cfl"] if p["rho_cfl"] > 0 else torch.zeros_like(r, dtype=torch.bool)
        solid = ~void

        def nb(w, ax, o):
            n = w.shape[ax]
            return w.index_select(ax, (torch.arange(n, device=w.device) + o).clamp(0, n - 1))

        def width(ax):
            n = r.shape[ax]
            k = torch.arange(n, device=r.device)
            shape = [1, 1, 1]
            shape[ax] = n
            return (1.0 + ((k > 0) & (k < n - 1)).to(r.dtype)).reshape(shape) * dx

        H = [width(a) for a in range(3)]
        L = [[(torch.where(nb(void, ax, 1), V[c], nb(V[c], ax, 1)) -
               torch.where(nb(void, ax, -1), V[c], nb(V[c], ax, -1))) / H[ax] for ax in range(3)] for c in range(3)]
        E = [[0.5 * (L[a][b] + L[b][a]) for b in range(3)] for a in range(3)]
        W = [[0.5 * (L[a][b] - L[b][a]) for b in range(3)] for a in range(3)]
        if p["axisym"]:
            E[1][1] = V[0] / self.rc
        tr = (E[0][0] + E[1][1] + E[2][2]) / 3
        S = [[s["Sxx"], s["Sxy"], s["Sxz"]], [s["Sxy"], s["Syy"], s["Syz"]], [s["Sxz"], s["Syz"], s["Szz"]]]
        name = [["Sxx", "Sxy", "Sxz"], ["Sxy", "Syy", "Syz"], ["Sxz", "Syz", "Szz"]]

        def adv(w):
            t = 0.0
            for ax in range(3):
                n = w.shape[ax]
                if n == 1:
                    continue
                up, dn = (w - nb(w, ax, -1)) / dx, (nb(w, ax, 1) - w) / dx
                t = t + V[ax] * torch.where(V[ax] > 0, up, dn)
            return t

        def put(k, x):
            d[k] = d[k] + torch.where(solid, x, torch.zeros_like(x))

        for a in range(3):
            for b in range(a, 3):
                J = sum(S[a][c] * W[c][b] - W[a][c] * S[c][b] for c in range(3))
                put(name[a][b], 2 * G * (E[a][b] - (tr if a == b else 0.0)) + J - adv(S[a][b]))
        put("D", -adv(s["D"]))
        put("vib", -adv(s["vib"]))
        for a, k in enumerate(("mu", "mv", "mw")):
            put(k, sum((nb(S[a][ax], ax, 1) - nb(S[a][ax], ax, -1)) / H[ax] for ax in range(3)))
        SV = [sum(S[ax][c] * V[c] for c in range(3)) for ax in range(3)]
        put("E", sum((nb(SV[ax], ax, 1) - nb(SV[ax], ax, -1)) / H[ax] for ax in range(3)))
        if p["axisym"]:
            put("mu", (S[0][0] - S[1][1]) / self.rc)
            put("mw", S[0][2] / self.rc)
            put("E", SV[0] / self.rc)
        if p["eta_af"] > 0:
            eta = torch.where(af > 0, af * p["eta_af"], torch.zeros_like(af))
            for c, k in enumerate(("mu", "mv", "mw")):
                lap = sum(nb(V[c], ax, 1) + nb(V[c], ax, -1) - 2 * V[c] for ax in range(3)) / (dx * dx)
                if p["axisym"] and c != 1:
                    lap = lap + L[c][0] / self.rc - (V[0] / self.rc ** 2 if c == 0 else 0.0)
                put(k, eta * lap)

    def clean(self, s):
        if not self.p["rho_cfl"] > 0:
            return
        bad = s["r"] < self.p["rho_cfl"]
        for k in ("mu", "mv", "mw") + (tuple(SPH_OUT_S) + ("E", "rc") if self.r0 is not None else ()):
            s[k] = torch.where(bad, torch.zeros_like(s[k]), s[k])
        if self.r0 is not None:
            s["r"] = torch.where(bad, self.r0, s["r"])

    def plastic(self, s, af):
        p = self.p
        if self.m["Y"] <= 0 and not p["rock"]:
            return
        if p["rock"]:
            P, c = self.pc(s)
            if p["af_prel"]:
                P = torch.where(s["vib"] > 0, torch.clamp(P - s["r"] * c * s["vib"], min=0), P)
            Yi = p["y_i0"] + p["mu_i"] * P / (1 + p["mu_i"] * P / max(p["y_m"] - p["y_i0"], 1.0))
            Yd = torch.clamp(p["y_d0"] + p["mu_d"] * P, max=p["y_m"])
            Y = (1 - s["D"]) * Yi + s["D"] * Yd
            if not p["af_prel"]:
                Y = Y * (1 - af)
        else:
            Y = (1 - s["D"]) * (1 - af) * self.m["Y"]
        J2 = 0.5 * (s["Sxx"] ** 2 + s["Syy"] ** 2 + s["Szz"] ** 2) + s["Sxy"] ** 2 + s["Sxz"] ** 2 + s["Syz"] ** 2
        vm = torch.sqrt(3 * J2)
        k = torch.where(vm > Y, Y / torch.clamp(vm, min=1e-300), torch.ones_like(Y))
        for q in SPH_OUT_S:
            s[q] = s[q] * k

    def damage(self, s, dt):
        m = self.m
        if m["Emod"] <= 0 or m["wk"] <= 0:
            return
        act = (1.0 / (m["wk"] * self.dx ** 3)) ** (1.0 / m["wm"])
        P, _ = self.pc(s)
        sig = torch.maximum(torch.maximum(s["Sxx"], s["Syy"]), s["Szz"]) - P
        grow = (sig > 0) & (sig / m["Emod"] > act) & (s["D"] < 1)
        d13 = s["D"] ** (1 / 3) + 0.4 * torch.sqrt(m["Emod"] / s["r"]) / (0.5 * self.dx) * dt
        s["D"] = torch.where(grow, torch.clamp(d13 ** 3, max=1.0), s["D"])

    def fluidize(self, s, dt):
        p = self.p
        if not (p["c_act"] > 0 and p["tdec"] > 0):
            return
        P, c = self.pc(s)
        dP = P - s["Pmax"]
        speed = torch.sqrt(s["mu"] ** 2 + s["mv"] ** 2 + s["mw"] ** 2) / s["r"]
        seed = dP / (s["r"] * c) if p["af_seeddp"] else speed
        hit = (dP > 0) & (dP > p["p_act"])
        s["vib"] = torch.where(hit, torch.maximum(s["vib"], p["c_act"] * seed), s["vib"]) * math.exp(-dt / p["tdec"])
        s["Pmax"] = torch.maximum(s["Pmax"], P)
        pv = s["r"] * c * s["vib"]
        s["af"] = pv / (pv + torch.clamp(P, min=p["p_coh"]))

    def adjust(self, s):
        gc = self.c
        if gc.pin_floor:
            k = gc.pin_floor
            s["r"][:, :, :k] = self.r0[:, :, :k]
            for q in ("mu", "mv", "mw", "E"):
                s[q][:, :, :k] = 0
        if gc.sponge_from >= 0:
            xi = torch.clamp(self.i - gc.sponge_from, min=0) / max(1, gc.shape[0] - 1 - gc.sponge_from)
            sp = xi * xi
            s["r"] = (1 - sp) * s["r"] + sp * self.r0
            for q in ("mu", "mv", "mw", "E"):
                s[q] = s[q] * (1 - sp)

    def run(self, steps):
        f, p = self.f, self.p
        for _ in range(steps):
            P, c = self.pc(f)
            c = torch.sqrt(c * c + (4.0 / 3.0) * self.m["G"] / f["r"]) if self.m["G"] > 0 else c
            sig = torch.sqrt(f["mu"] ** 2 + f["mv"] ** 2 + f["mw"] ** 2) / f["r"] + c
            dt = self.c.cfl * self.dx / float(sig[f["r"] >= p["rho_cfl"]].max())
            self.fluidize(f, dt)
            d = self.lop(f, f["af"])
            g = {k: f[k] + dt * d[k] if k in d else f[k] for k in f}
            self.clean(g)
            self.plastic(g, f["af"])
            d = self.lop(g, f["af"])
            for k in d:
                f[k] = 0.5 * (f[k] + g[k] + dt * d[k])
            self.damage(f, dt)
            self.plastic(f, f["af"])
            self.clean(f)
            self.adjust(f)
        return f
