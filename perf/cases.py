"""Performance cases of the framework: the work a time step of a marker-in-cell
Stokes model asks of it, over the sizes that the configurations, tests and
benchmark use (33^3 to 257^3 nodes, 1 to 20 spheres or a layered lithosphere).

Kinds:
  solve   new node fields in, velocities and pressure out (p2_set_nodes and
          p2_stokes_solve, what vpiterate() asks for on every step)
  batch   independent instances of uneven sizes solved at once
          (p2_stokes_solve_batch)
  nodes   marker -> node interpolation of resident markers, fields read back
  scratch marker -> node interpolation on device arrays without allocation
  move    fourth-order Runge-Kutta marker advection on host arrays
  heat    one heat-equation step with markers on host arrays

Solves run to a relative residual of `tol`.  The usual target is 1e-8; a solve
here asks for more (a program that differentiates the pressure does, too), so
that the answers of two builds agree to the last digits their types promise
instead of stopping at different places of the same convergence history.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import pardiso2_b200 as P
from pardiso2_b200 import capi, model as M

FIELDS = ("nu", "ro", "nxx", "nxy", "nxz", "nyz")


def _solve(name, shape, precision, spheres, tol, contrast=2.0, smoother=1, growth=1, sweeps=4, restart=16):
    d = {"kind": "solve", "nx": shape[0], "ny": shape[1], "nz": shape[2], "precision": precision,
         "spheres": spheres, "contrast": contrast, "tol": tol, "smoother": smoother, "growth": growth,
         "sweeps": sweeps, "restart": restart}
    return dict(d, name=name) if name else d


def listed():
    return [
        # the plain method's grid, one inclusion: the smallest solve, all latency
        _solve("solve33_mixed", (33, 33, 33), "mixed", 1, 1e-11),
        # the same grid in FP64 throughout, odd and uneven sides
        _solve("solve37x33x41_fp64", (37, 33, 41), "fp64", 3, 1e-11),
        # the everyday model: 65^3, eight inclusions, both precisions
        _solve("solve65_mixed", (65, 65, 65), "mixed", 8, 1e-11, contrast=3.0, restart=12),
        _solve("solve65_fp64", (65, 65, 65), "fp64", 8, 1e-11, contrast=3.0),
        # uneven sides, none of them a power of two plus one
        _solve("solve91x97x79_mixed", (91, 97, 79), "mixed", 5, 1e-11),
        # many inclusions: the diagonal cell block with doubling sweeps
        _solve("solve129_mixed", (129, 129, 129), "mixed", 20, 1e-10, smoother=0, growth=2),
        # the layered lithosphere at 257^3 (68 M unknowns), the headline model
        _solve("layered257_mixed", (257, 257, 257), "mixed", 0, 1e-10, contrast=4.0, growth=2, sweeps=2),
        # parameter study: independent models of uneven sizes at once
        {"name": "batch8", "kind": "batch", "sizes": "33,49,65,33,81,49,65,33", "tol": 1e-12},
        # a host code with its own device arrays and no allocations: the smallest call
        {"name": "scratch21", "kind": "scratch", "nx": 21, "ny": 21, "nz": 21, "per_axis": 3},
        # resident markers of the 129^3 model
        {"name": "nodes129", "kind": "nodes", "nx": 129, "ny": 129, "nz": 129, "per_axis": 2},
        # marker advection of the 65^3 model through the host-array call
        {"name": "move65", "kind": "move", "nx": 65, "ny": 65, "nz": 65, "per_axis": 2},
        # heat step of the 65^3 model, all heating terms and the markers
        {"name": "heat65", "kind": "heat", "nx": 65, "ny": 65, "nz": 65, "per_axis": 2},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, lo, hi):
    # odd node counts: the reference's coarsening rule leaves a coarse line without weight on even ones
    n = _log(rng, lo, hi)
    return tuple(max(33, min(257, int(round(n * rng.uniform(0.85, 1.15))))) // 2 * 2 + 1 for _ in range(3))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["batch", "scratch", "nodes", "move", "heat"])
    if kind == "solve":
        smoother = rng.choice([1, 1, 0])
        return _solve(None, _sides(rng, 33, 180), rng.choice(["mixed", "mixed", "fp64"]), rng.randint(1, 10), 1e-11,
                      contrast=rng.uniform(1.0, 2.0), smoother=smoother,
                      growth=2 if smoother == 0 else rng.choice([1, 2]), sweeps=4, restart=rng.choice([12, 16]))
    if kind == "batch":
        sizes = [rng.choice([33, 49, 65, 81, 97]) for _ in range(rng.randint(2, 8))]
        return {"kind": "batch", "sizes": ",".join(map(str, sizes)), "tol": 1e-12}
    if kind == "scratch":
        n = [rng.randint(9, 40) for _ in range(3)]
        return {"kind": "scratch", "nx": n[0], "ny": n[1], "nz": n[2], "per_axis": rng.randint(1, 2)}
    hi = {"nodes": 160, "move": 129, "heat": 97}[kind]
    s = _sides(rng, 33, hi)
    return {"kind": kind, "nx": s[0], "ny": s[1], "nz": s[2], "per_axis": rng.randint(1, 2)}


# ---------------------------------------------------------------------------
# Models


def _multinum(shape):
    """Levels as the configurations have them: coarsen while every side keeps nine nodes."""
    n, m = min(shape), 0
    while (n - 5) // 2 + 5 >= 9:
        n, m = (n - 5) // 2 + 5, m + 1
    return m


@functools.lru_cache(maxsize=16)
def _box(shape, thermal=False):
    """Grid lines, levels and boundary tables of a closed free-slip unit box, the same for every model on it."""
    g = [M.uniform_lines(n) for n in shape]
    lv = M.make_levels(*g, _multinum(shape))
    sp = M.SolverParams()
    lines = M.free_slip_lines(sp.pin, sp.pinit)
    return g, lv, M.build_bc_tables(lv, lines + M.thermal_lines() if thermal else lines)


def _model(shape, nubeg=1e-6, nuend=1e8, thermal=False):
    g, lv, bc = _box(shape, thermal)
    none = np.zeros(0, np.float32)
    rocks = M.Rocks(np.ones(1), np.ones(1), np.zeros(1))
    return M.Model("box", *g, lv.multinum, lv, bc, none, none, none, np.zeros(0, np.int8), rocks,
                   M.SolverParams(nubeg=nubeg, nuend=nuend))


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _gen(seed):
    return torch.Generator().manual_seed(int(seed))


def _spheres(count, contrast, gen):
    """centre, radius, viscosity (log-uniform in 10^+-contrast), density per sphere, as plain numbers"""
    u = torch.rand((count, 6), generator=gen, dtype=torch.float64)
    top = 0.12 if count > 1 else 0.2
    return [(*(0.15 + 0.7 * r[:3]).tolist(), 0.05 + (top - 0.05) * r[3].item(),
             10.0 ** (contrast * (2 * r[4].item() - 1)), 2 * r[5].item() - 1) for r in u]


def _rock(x, y, z, case, spheres, jitter):
    """viscosity and density at points (broadcast coordinates)"""
    if case.get("spheres", 1) == 0:
        # layered lithosphere: exp(-ln(1e4) z) from 1e4 down to 1, a dense slab, a weak zone
        nu = torch.exp(math.log(10.0) * case["contrast"] * (1 - z)) + 0 * x + 0 * y
        ro = torch.zeros_like(nu)
        slab = ((x - 0.45 - jitter[0]).abs() <= 0.1) & ((y - 0.5).abs() <= 0.3) & ((z - 0.625).abs() <= 0.175)
        weak = ((x - 0.775).abs() <= 0.075) & ((y - 0.5).abs() <= 0.3) & (z >= 0.55 + jitter[1])
        nu = torch.where(slab, torch.full_like(nu, 1e3), torch.where(weak, torch.full_like(nu, 1e-2), nu))
        return nu, torch.where(slab, torch.full_like(ro, 1.0 + jitter[2]), ro)
    nu = torch.ones_like(x + y + z)
    ro = torch.zeros_like(nu)
    for cx, cy, cz, rad, eta, rho in spheres:
        inside = (x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2 <= rad * rad
        nu = torch.where(inside, torch.full_like(nu, eta), nu)
        ro = torch.where(inside, torch.full_like(ro, rho), ro)
    return nu, ro


def _fields(case, seed):
    """Node fields of a seeded model, averaged over the eight markers around
    each position: nu, ro at the nodes, nxx at cell centres, nxy .. nyz on edges."""
    gen = _gen(seed)
    nx, ny, nz = _shape(case)
    sph = _spheres(max(1, case["spheres"]), case["contrast"], gen)
    jitter = ((torch.rand(3, generator=gen, dtype=torch.float64) - 0.5) * 0.1).tolist()
    h = 1.0 / (nx - 1), 1.0 / (ny - 1), 1.0 / (nz - 1)
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") * s for n, s in zip((nx, ny, nz), h)]
    out = {}
    for key, off in (("node", (0, 0, 0)), ("nxx", (-.5, -.5, -.5)), ("nxy", (0, 0, .5)), ("nxz", (0, .5, 0)),
                     ("nyz", (.5, 0, 0))):
        nu, ro = 0, 0
        for q in range(8):
            s = [off[a] + (0.25 if q >> a & 1 else -0.25) for a in range(3)]
            x, y, z = (ax[a] + s[a] * h[a] for a in range(3))
            v, r = _rock(x[None, :, None], y[None, None, :], z[:, None, None], case, sph, jitter)
            nu, ro = nu + v.float() / 8, ro + r.float() / 8
        if key == "node":
            out["nu"], out["ro"] = nu, ro
        else:
            out[key] = nu
    pinned = {}
    for k in FIELDS:
        pinned[k] = torch.empty(nx * ny * nz, dtype=torch.float32, pin_memory=True)
        pinned[k].copy_(out[k].reshape(-1))
    return pinned


def _problem(m, precision, tol, smoother=1, growth=1, sweeps=4, restart=16):
    nl = m.multinum + 1
    per = [sweeps] + [min(64, 4 * growth ** l) for l in range(1, nl)]
    return P.StokesProblem(m, precision=precision, tol=tol, npre=per, npost=per, restart=restart, max_iter=400,
                           smoother=smoother)


def _markers(shape, per_axis, seed):
    """Jittered markers, per_axis per cell and axis, cell by cell, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    cells = [n - 1 for n in shape]
    p = per_axis
    out = []
    for a in range(3):
        sub = (torch.arange(p, device="cuda", dtype=torch.float64) + 0.5) / p
        line = (torch.arange(cells[a], device="cuda", dtype=torch.float64)[:, None] + sub) / cells[a]
        # order: cell z, x, y, then within the cell z, x, y
        at = {2: (0, 3), 0: (1, 4), 1: (2, 5)}[a]
        view = [1] * 6
        view[at[0]], view[at[1]] = cells[a], p
        full = line.reshape(view).expand(cells[2], cells[0], cells[1], p, p, p).reshape(-1)
        full = full + (torch.rand(full.numel(), generator=gen, device="cuda", dtype=torch.float64) - 0.5) / (p * cells[a])
        out.append(full.float())
    typ = ((out[0] - 0.5) ** 2 + (out[1] - 0.5) ** 2 + (out[2] - 0.5) ** 2 < 0.04).to(torch.int8)
    typ += 2 * (out[2] > 0.8).to(torch.int8)
    return out + [typ]


ROCK_NU = np.array([1.0, 1e3, 10.0, 1e2])
ROCK_RO = np.array([0.0, 1.0, -0.5, 0.25])


def _pin(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p


def _at(t):
    return t.data_ptr()


# ---------------------------------------------------------------------------
# Preparation: what the program holds before the call


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_solve(case, seed):
    f = _fields(case, seed)
    lo, hi = float(f["nu"].min()), float(f["nu"].max())
    m = _model(_shape(case), nubeg=0.5 * min(1.0, lo), nuend=2 * max(1.0, hi))
    prob = _problem(m, 1 if case["precision"] == "fp64" else 0, case["tol"], case["smoother"], case["growth"],
                    case["sweeps"], case["restart"])
    n = m.nodenum
    sol = {k: torch.zeros(n, dtype=torch.float64 if k == "pr" else torch.float32, pin_memory=True)
           for k in ("vx", "vy", "vz", "pr")}
    return {"kind": "solve", "prob": prob, "fields": {k: v.numpy() for k, v in f.items()}, "keep": f, "sol": sol,
            "host": {k: v.numpy() for k, v in sol.items()}}


def _run_solve(s):
    for v in s["sol"].values():
        v.zero_()  # from rest
    s["prob"].set_nodes(s["fields"])
    s["prob"].vpiterate(**s["host"])
    return s["sol"]


def _prepare_batch(case, seed):
    probs, sols = [], []
    for i, n in enumerate(int(v) for v in case["sizes"].split(",")):
        sub = {"nx": n, "ny": n, "nz": n, "spheres": 1 + (seed + 3 * i) % 10, "contrast": 2.0}
        f = _fields(sub, seed * 1000 + i)
        m = _model((n, n, n), nubeg=0.5 * min(1.0, float(f["nu"].min())), nuend=2 * max(1.0, float(f["nu"].max())))
        prob = _problem(m, 0, case["tol"])
        prob.set_nodes({k: v.numpy() for k, v in f.items()})
        probs.append(prob)
        sols.append({k: torch.zeros(n ** 3, dtype=torch.float64, pin_memory=True) for k in ("vx", "vy", "vz", "pr")})
    return {"kind": "batch", "probs": probs, "sols": sols}


def _run_batch(s):
    capi.solve_batch([p.ctx for p in s["probs"]])
    for p, o in zip(s["probs"], s["sols"]):
        p.ctx._check(p.ctx.L.p2_get_solution(p.ctx.h, _at(o["vx"]), _at(o["vy"]), _at(o["vz"]), _at(o["pr"])), "get")
    return s["sols"]


def _scratch_call():
    f = capi.load().p2_ronurecalc_noalloc
    vp = C.c_void_p
    f.argtypes = ([C.c_int] * 3 + [vp] * 3 + [C.POINTER(capi.Params), C.c_int] + [vp] * 3 + [C.c_long] + [vp] * 4
                  + [vp] * 6 + [vp, C.c_char_p, C.c_long])
    f.restype = C.c_int
    return f


def _prepare_scratch(case, seed):
    shape = _shape(case)
    g = [M.uniform_lines(n) for n in shape]
    prm = P.default_params()
    prm.nubeg, prm.nuend = 0.5, 2e3
    n = shape[0] * shape[1] * shape[2]
    return {"kind": "scratch", "call": _scratch_call(), "g": g, "prm": prm, "n": shape,
            "mk": _markers(shape, case["per_axis"], seed),
            "out": [torch.ones(n, dtype=torch.float32, device="cuda") for _ in FIELDS],
            "stream": torch.cuda.current_stream().cuda_stream, "err": C.create_string_buffer(256)}


def _run_scratch(s):
    nx, ny, nz = s["n"]
    mk = s["mk"]
    st = s["call"](nx, ny, nz, *[a.ctypes.data for a in s["g"]], C.byref(s["prm"]), len(ROCK_NU),
                   ROCK_NU.ctypes.data, ROCK_NU.ctypes.data, ROCK_RO.ctypes.data, mk[0].numel(), *map(_at, mk),
                   *map(_at, s["out"]), s["stream"], s["err"], len(s["err"]))
    if st:
        raise RuntimeError(s["err"].value.decode())
    return dict(zip(FIELDS, s["out"]))


def _prepare_nodes(case, seed):
    m = _model(_shape(case), nubeg=0.5, nuend=2e3)
    ctx = P.Context(0)
    ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m))
    mk = [t.cpu().numpy() for t in _markers(_shape(case), case["per_axis"], seed)]
    ctx.upload_markers(*mk, ROCK_NU, ROCK_NU, ROCK_RO)
    return {"kind": "nodes", "ctx": ctx,
            "out": {k: torch.zeros(m.nodenum, dtype=torch.float32, pin_memory=True) for k in FIELDS}}


def _run_nodes(s):
    s["ctx"].ronurecalc_resident()
    s["ctx"]._check(s["ctx"].L.p2_get_nodes(s["ctx"].h, *[_at(s["out"][k]) for k in FIELDS]), "p2_get_nodes")
    return s["out"]


def _velocity(shape, seed):
    """a smooth closed-box velocity, about one cell per unit time"""
    gen = _gen(seed)
    a = torch.rand(6, generator=gen, dtype=torch.float64).tolist()
    ax = [torch.linspace(0, 1, n, dtype=torch.float64, device="cuda") for n in shape]
    x, y, z = ax[0][None, :, None], ax[1][None, None, :], ax[2][:, None, None]
    pi = math.pi
    v = [torch.sin(pi * x) * torch.cos(pi * y * (1 + a[0])) * torch.cos(pi * z * (1 + a[1])),
         torch.cos(pi * x * (1 + a[2])) * torch.sin(pi * y) * torch.cos(pi * z * (1 + a[3])),
         torch.cos(pi * x * (1 + a[4])) * torch.cos(pi * y * (1 + a[5])) * torch.sin(pi * z)]
    return [(t / max(shape)).float().reshape(-1) for t in v]


def _prepare_move(case, seed):
    m = _model(_shape(case))
    ctx = P.Context(0)
    ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m))
    mk = [_pin(t) for t in _markers(_shape(case), case["per_axis"], seed)]
    return {"kind": "move", "ctx": ctx, "vel": [_pin(t) for t in _velocity(_shape(case), seed + 1)], "mk": mk,
            "pos": [torch.empty_like(t, pin_memory=True) for t in mk[:3]]}


def _run_move(s):
    for o, t in zip(s["pos"], s["mk"]):
        o.copy_(t)  # the call moves the markers in place
    L = s["ctx"].L
    s["ctx"]._check(L.p2_movemark(s["ctx"].h, 0.5, 2, 0, *[v.numpy() for v in s["vel"]], s["pos"][0].numel(),
                                  *[p.numpy() for p in s["pos"]], s["mk"][3].numpy()), "p2_movemark")
    return s["pos"]


def _prepare_heat(case, seed):
    shape = _shape(case)
    m = _model(shape, thermal=True)
    ctx = P.Context(0)
    ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m))
    ctx.heat_set_bc(m.bc, m.nodenum)
    th = M.thermal_fields(m, seed=seed, heat=(2e4, 8e4))
    nt = m.multinum
    hp = capi.heat_params(maxtkstep=25.0, heatmin=2e-3, heatdif=1.0, multinumt=nt, multicyct=1, pre=[3] * nt + [0],
                          post=[0] + [3] * (nt - 1) + [10], frictyn=1, adiabyn=1, max_cycles=200)
    mk = [t.cpu().numpy() for t in _markers(shape, case["per_axis"], seed)]
    gen = _gen(seed + 2)
    se = [(2 * torch.rand(m.nodenum, generator=gen) - 1).numpy() for _ in range(12)]
    return {"kind": "heat", "ctx": ctx, "hp": hp, "th": th, "vel": [v.cpu().numpy() for v in _velocity(shape, seed)],
            "se": se, "mk": mk, "tk": np.full(len(mk[0]), 900.0, np.float32),
            "dt": 2000.0 * (64.0 / (max(shape) - 1)) ** 2}


def _run_heat(s):
    tk, mk, info = s["ctx"].titerate(s["hp"], s["dt"], s["th"], vel=s["vel"], se=s["se"], markers=s["mk"],
                                     markk=s["tk"])
    return {"tk": tk, "markk": mk, "substeps": info.substeps}


# ---------------------------------------------------------------------------
# The interpolations in 64 bits


def exact(case, seed):
    """run()'s answer in 64 bits.  None for the solves (a 64-bit factorisation of 144 thousand to 68 million
    unknowns takes minutes and more) and the heat step (an iteration to its own error bound on stored 32-bit
    temperatures)."""
    if case["kind"] in ("scratch", "nodes"):
        old = 1.0 if case["kind"] == "scratch" else 0.0
        return _exact_nodes(case, seed, old)
    if case["kind"] == "move":
        return _exact_move(case, seed)
    return None


def _lines(n):
    return torch.cumsum(torch.full((n,), 1.0 / (n - 1), dtype=torch.float64, device="cuda"), 0) - 1.0 / (n - 1)


def _exact_nodes(case, seed, old):
    shape = _shape(case)
    n = shape[0] * shape[1] * shape[2]
    mk = _markers(shape, case["per_axis"], seed)
    g = [_lines(k) for k in shape]
    inside = torch.ones_like(mk[0], dtype=torch.bool)
    for a in range(3):
        inside &= (mk[a] > 0) & (mk[a].double() < g[a][-1])
    pos = [t[inside].double() for t in mk[:3]]
    typ = mk[3][inside].long()
    eta, rho = (torch.tensor(t, device="cuda")[typ] for t in (ROCK_NU, ROCK_RO))
    cell = [(torch.searchsorted(g[a], pos[a], right=True) - 1).clamp(0, shape[a] - 2) for a in range(3)]
    top = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k in FIELDS}
    low = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k in FIELDS}

    def add(key, node, weight, value, where):
        w = torch.where(where, weight, torch.zeros_like(weight))
        top[key].index_add_(0, node, w * value)
        low[key].index_add_(0, node, w)

    for q in range(8):
        up = [q >> a & 1 for a in range(3)]
        idx = [cell[a] + up[a] for a in range(3)]
        node = (idx[2] * shape[0] + idx[0]) * shape[1] + idx[1]
        d = [1 - (g[a][idx[a]] - pos[a]).abs() / (g[a][cell[a] + 1] - g[a][cell[a]]) for a in range(3)]
        near = [t > 0.5 for t in d]
        half = [t - 0.5 for t in d]
        mid = [0.5 - t.abs() for t in half]
        add("nu", node, d[0] * d[1] * d[2], eta, (d[0] > 0) & (d[1] > 0) & (d[2] > 0))
        if all(up):
            add("nxx", node, 8 * mid[0] * mid[1] * mid[2], eta, near[0] | True)
        if not up[2]:
            add("nxy", node, 8 * half[0] * half[1] * mid[2], eta, near[0] & near[1])
        if not up[1]:
            add("nxz", node, 8 * half[0] * mid[1] * half[2], eta, near[0] & near[2])
        if not up[0]:
            add("nyz", node, 8 * mid[0] * half[1] * half[2], eta, near[1] & near[2])
        add("ro", node, 8 * half[0] * half[1] * half[2], rho, near[0] & near[1] & near[2])
    out = {}
    for k in FIELDS:
        v = torch.where(low[k] > 0, top[k] / low[k], torch.full_like(low[k], old))
        out[k] = (v if k == "ro" else v.clamp(0.5, 2e3)).cpu()
    return out


def _exact_move(case, seed):
    shape = _shape(case)
    mk = _markers(shape, case["per_axis"], seed)
    vel = [v.double() for v in _velocity(shape, seed + 1)]
    g = [_lines(k) for k in shape]

    def axis(a, x, aligned):
        n, line = shape[a], g[a]
        cell = (torch.searchsorted(line, x, right=True) - 1).clamp(0, n - 2)
        if aligned:
            lo, x0, x1 = cell, line[cell], line[cell + 1]
        else:
            mid = 0.5 * (line[1:] + line[:-1])
            lo = (cell - (x < mid[cell]).long()).clamp(0, n - 3)
            x0, x1 = mid[lo], mid[lo + 1]
            x = torch.minimum(torch.maximum(x, mid[0]), mid[n - 2])
        w1 = (x - x0) / (x1 - x0)
        return lo, (1 - w1, w1)

    def at(p):
        p = [p[a].clamp(0, 1) for a in range(3)]
        out = []
        for comp in range(3):
            ax = [axis(a, p[a], a == comp) for a in range(3)]
            s = 0
            for q in range(8):
                up = [q >> a & 1 for a in range(3)]
                node = ((ax[2][0] + up[2]) * shape[0] + ax[0][0] + up[0]) * shape[1] + ax[1][0] + up[1]
                s = s + vel[comp][node] * ax[0][1][up[0]] * ax[1][1][up[1]] * ax[2][1][up[2]]
            out.append(s)
        return out

    p0, dt = [t.double() for t in mk[:3]], 0.5
    k1 = at(p0)
    k2 = at([p + dt / 2 * k for p, k in zip(p0, k1)])
    k3 = at([p + dt / 2 * k for p, k in zip(p0, k2)])
    k4 = at([p + dt * k for p, k in zip(p0, k3)])
    return [(p + dt * (a + 2 * b + 2 * c + d) / 6).cpu() for p, a, b, c, d in zip(p0, k1, k2, k3, k4)]


# ---------------------------------------------------------------------------
# What a pass cannot do without


def work(case):
    """Bytes in and out of one pass, each once; the arithmetic of the discretisation for a solve's answer (one
    operator application per unknown) or of the interpolations."""
    if case["kind"] == "batch":
        n = sum(int(v) ** 3 for v in case["sizes"].split(","))
        return {"bytes": 56.0 * n, "flops": 400.0 * n}
    nx, ny, nz = _shape(case)
    n = nx * ny * nz
    if case["kind"] == "solve":
        # six float fields in, three float velocities and a double pressure in and out
        return {"bytes": (24 + 20 + 20) * float(n), "flops": 400.0 * n}
    mk = (nx - 1) * (ny - 1) * (nz - 1) * case["per_axis"] ** 3
    if case["kind"] in ("scratch", "nodes"):
        return {"bytes": 13.0 * mk + 24 * n, "flops": 8 * 30.0 * mk}
    if case["kind"] == "move":
        return {"bytes": 25.0 * mk + 12 * n, "flops": 4 * 100.0 * mk}
    # heat: six fields and twelve stress / strain-rate fields in, temperature out; markers with their temperature
    return {"bytes": (24 + 12 + 48 + 4) * float(n) + 21.0 * mk, "flops": 100.0 * n + 100.0 * mk}
