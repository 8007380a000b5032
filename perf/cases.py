"""Performance cases: the calls of a time step, through the package's public entry points.

Kinds of case:
  project   one projection of a face velocity field (B200PressureSolver.project) with the coefficients of a
            single-phase box, a two-phase sphere or a box with solid spheres already installed
  pressure  the implicit half of a time step (SMACStep): solve_poisson with new coefficients, correct_vof_velocity,
            update_boundary_ghost, make_face_gradp
  adjoint   a differentiable projection, forward and backward (autograd.project)
  explicit  the explicit half of a time step (SMACStep): properties, mass flux, outlet coefficients, surface
            tension, predictor, wall u*
  predict   the momentum predictor alone (SMACStep.get_vof_vstar_rhouu_consistent)

Inputs come from a seeded generator on the GPU.  exact() restates every call in plain torch at 64 bits.
"""
import math

import numpy as np
import torch

from mydemcfd_b200 import _native as nat
from mydemcfd_b200 import autograd as ag
from mydemcfd_b200.solver import B200PressureSolver, BoundaryConditions, DeviceGrid, SMACStep

DEV = "cuda"
F64, U8 = torch.float64, torch.uint8
RHO0, MU0, MU1 = 1.0, 1e-3, 1e-1
SIGMA = 0.07
GRAVITY = (0.0, 0.0, -9.8)
# boundary ids of the cases: 0 no-slip wall, 1 outlet, 2 inflow with velocity (1, 0, 0)
BC_TYPE = (0, 4, 2)
BC_V = ((0.0, 0.0, 1.0), (0.0, 0.0, 0.0), (0.0, 0.0, 0.0))


# ---------------------------------------------------------------------------
# the cases
def _case(kind, nx, ny, nz, **kw):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "mixed": False, "fluid": "plain", "ratio": 1.0, "spheres": 0,
         "channel": False, "coupled": False}
    c.update(kw)
    return c


def listed():
    cs = [
        # the smallest projection: a debugging run or a unit test; launches and host round trips count
        _case("project", 32, 32, 32, name="project_32_fp64"),
        # a small production run in mixed precision
        _case("project", 64, 64, 64, mixed=True, name="project_64_mixed"),
        # the benchmark workload, in both precisions
        _case("project", 256, 256, 256, mixed=True, name="project_256_mixed"),
        _case("project", 256, 256, 256, name="project_256_fp64"),
        # a decimal grid around solid spheres (a packed bed): the extents halve only once or twice
        _case("project", 150, 100, 75, mixed=True, fluid="ibm", spheres=40, name="project_ibm_150x100x75_mixed"),
        # the implicit half of a two-phase step, coefficients new each step (the 1000:1 sphere workload)
        _case("pressure", 192, 192, 192, mixed=True, fluid="vof", ratio=1000.0, name="pressure_vof_192_mixed"),
        # the same in FP64 in a channel with inflow and outlet, ragged rows
        _case("pressure", 200, 100, 72, fluid="vof", ratio=100.0, channel=True,
              name="pressure_channel_200x100x72_fp64"),
        # training through the solver: forward and backward (the 128^3 adjoint workload)
        _case("adjoint", 128, 128, 128, mixed=True, fluid="vof", ratio=100.0, name="adjoint_vof_128_mixed"),
        # the explicit half of the two-phase step
        _case("explicit", 192, 192, 192, fluid="vof", ratio=1000.0, name="explicit_vof_192"),
        # the smallest explicit half, odd extents, solids: launch bound
        _case("explicit", 45, 37, 41, fluid="vof", ratio=1000.0, spheres=2, name="explicit_ibm_45x37x41"),
        # the coupled (two-way) explicit half in a channel with particles, odd extents
        _case("explicit", 161, 95, 130, fluid="vof", ratio=1000.0, coupled=True, channel=True,
              name="explicit_coupled_161x95x130"),
        # the predictor alone on the benchmark grid, the largest explicit call of a step
        _case("predict", 256, 256, 256, fluid="vof", ratio=1000.0, name="predict_256"),
    ]
    return cs


def _halved(n):
    """An extent after halving while it is even and its half at least 4."""
    while n % 2 == 0 and n // 2 >= 4:
        n //= 2
    return n


def draw(rng):
    kind = rng.choice(("project", "project", "pressure", "adjoint", "explicit", "explicit", "predict"))
    implicit = kind in ("project", "pressure", "adjoint")
    while True:
        n = [int(round(math.exp(rng.uniform(math.log(20), math.log(256))))) for _ in range(3)]
        if implicit:                # extents of which some halve, as users choose them
            n = [m if rng.random() < 0.3 else (m // 4 * 4 if rng.random() < 0.5 else m // 16 * 16) for m in n]
            if min(n) < 16 or math.prod(_halved(m) for m in n) > 60000:
                continue
        if n[0] * n[1] * n[2] <= 192 ** 3 and max(n) <= 8 * min(n):
            break
    fluid = rng.choice(("plain", "vof", "ibm")) if kind == "project" else "vof"
    ratio = rng.choice((10.0, 100.0, 1000.0)) if fluid == "vof" else 1.0
    nsph = rng.randint(1, 20) if fluid == "ibm" else rng.choice((0, 0, 3)) if kind in ("explicit", "predict") else 0
    return _case(kind, *n, mixed=kind in ("project", "pressure", "adjoint") and rng.random() < 0.6, fluid=fluid,
                 ratio=ratio, spheres=nsph, channel=kind in ("pressure", "explicit", "predict") and rng.random() < 0.4,
                 coupled=kind in ("pressure", "explicit", "predict") and rng.random() < 0.4)


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    k = case["kind"]
    types = 4                       # one cell and three face types
    if k == "project":              # u*, f_b, types in; p_delta, u out
        b, f = 3 * 8 + 3 * 8 + types + 8 + 3 * 8, 60
    elif k == "pressure":           # u*, f_b, f_inv_rho, f_s, rho, types, ids in; p, p_delta, rhs, u, grad p out
        b, f = 4 * 24 + 8 + types + 3 + 3 * 8 + 2 * 24 + (16 if case["coupled"] else 0), 80
    elif k == "adjoint":            # alpha, u*, dL/du, types in; u, p_delta, dL/du* out
        b, f = 8 + 2 * 24 + types + 24 + 8 + 24, 120
    else:
        # predictor: u, mf, mu_f, f_b on faces, mu, rho_old, p, types, ids in; u* out
        b, f = 4 * 24 + 3 * 8 + types + 3 + 24, 200
        if case["coupled"]:
            b += 24 + 2 * 8         # impulse, two void fractions
        if case["spheres"]:
            b += 2 * 24             # solid fractions of the faces
        if k == "explicit":
            # alpha, F in; rho, 1/rho, mu, rho_f, f_inv_rho (f_b, mu_f, mf counted), n, kappa, |grad|, f_s out
            b += 8 + 24 + 3 * 8 + 4 * 24 + 24 + 5 * 8 + 24
            f += 150
    return {"bytes": float(b * n), "flops": float(f * n)}


def tolerance(case):
    if case["kind"] in ("explicit", "predict"):
        return {"rel": 1e-12, "max": 1e-10}
    # a solve to a relative residual of 1e-8: the pressure's error is that times what the operator's spectrum
    # makes of it: up to 1.2e-6 from exact() (and 5.8e-6 at one value) over the listed and 30 drawn cases
    return {"rel": 5e-6, "max": 5e-5}


# ---------------------------------------------------------------------------
# inputs (plain torch; arrays (sz, sy, sx), x fastest; axis 0 is x)
def _n(case):
    return (case["nx"], case["ny"], case["nz"])


def _shape(n, fam=None):
    s = [n[0] + 2, n[1] + 2, n[2] + 2]
    if fam is not None:
        s[fam] += 1
    return (s[2], s[1], s[0])


def _sl(a, ax, lo, hi):
    return a.narrow(2 - ax, lo, hi - lo)


def _rand(gen, shape, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=gen, dtype=F64, device=DEV).mul_(hi - lo).add_(lo)


def _coords(n, h, fam=None):
    """Coordinates of cell centres, or of the faces of a family, as three broadcastable tensors (x, y, z)."""
    out = []
    for ax in range(3):
        s = n[ax] + 2 + (1 if fam == ax else 0)
        c = (torch.arange(s, dtype=F64, device=DEV) - (1.0 if fam == ax else 0.5)) * h[ax]
        shp = [1, 1, 1]
        shp[2 - ax] = s
        out.append(c.reshape(shp))
    return out


def _radius(n, h, centre, fam=None):
    x, y, z = _coords(n, h, fam)
    return torch.sqrt((x - centre[0]) ** 2 + (y - centre[1]) ** 2 + (z - centre[2]) ** 2)


def _spheres(case, h, seed):
    """Non-overlapping spheres inside the box: radii of a twentieth to a seventh of the smallest extent."""
    rng = np.random.default_rng(seed + 77)
    ext = np.array(_n(case)) * np.array(h)
    out = []
    for _ in range(20000):
        if len(out) >= case["spheres"]:
            break
        r = rng.uniform(0.05, 0.14) * ext.min()
        lo = r + 2.5 * max(h)
        c = lo + (ext - 2 * lo) * rng.random(3)
        if all(np.linalg.norm(c - o[:3]) > r + o[3] + 2.5 * max(h) for o in out):
            out.append(np.append(c, r))
    return out


def _base(case, seed):
    """Types, ids, marks, volume fraction and solids of a case."""
    n = _n(case)
    h = (1.0 / n[0],) * 3
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1000003 * seed + 7)
    ct = torch.full(_shape(n), 2, dtype=U8, device=DEV)
    ct[1:-1, 1:-1, 1:-1] = 0
    ft, bid, marks = [], [], []
    for fam in range(3):
        t = torch.full(_shape(n, fam), 2, dtype=U8, device=DEV)
        v = t
        for ax in range(3):
            v = _sl(v, ax, 1, n[ax] + 1 + (1 if ax == fam else 0))
        v.fill_(0)
        for i in (0, n[fam]):
            _sl(v, fam, i, i + 1).fill_(1)
        ft.append(t)
        bid.append(torch.zeros_like(t))
        marks.append(torch.zeros_like(t))
    if case["channel"]:
        bid[0][1:-1, 1:-1, 1] = 2
        bid[0][1:-1, 1:-1, n[0] + 1] = 1
        marks[0][1:-1, 1:-1, n[0] + 1] = 2
    B = {"n": n, "h": h, "gen": gen, "ct": ct, "ft": ft, "bid": bid, "marks": marks if case["channel"] else None}
    ext = [n[k] * h[k] for k in range(3)]
    rng = np.random.default_rng(seed)
    if case["fluid"] == "vof":
        centre = [(0.3 + 0.4 * rng.random()) * e for e in ext]
        B["alpha"] = (0.5 - (_radius(n, h, centre) - 0.25 * min(ext)) / (1.5 * h[0])).clamp_(0.0, 1.0)
    B["sf"] = None
    if case["spheres"]:
        sph = _spheres(case, h, seed)
        solid = torch.zeros(_shape(n), dtype=torch.bool, device=DEV)
        sf = [torch.zeros(_shape(n, f), dtype=F64, device=DEV) for f in range(3)]
        for s in sph:
            solid |= _radius(n, h, s) < s[3]
            for f in range(3):
                torch.maximum(sf[f], (0.5 - (_radius(n, h, s, f) - s[3]) / h[0]).clamp_(0.0, 1.0), out=sf[f])
        ct[solid] = 3
        for f in range(3):
            _sl(ft[f], f, 0, n[f] + 2)[solid] = 1
            _sl(ft[f], f, 1, n[f] + 3)[solid] = 1
        B["sf"] = sf
    return B


def _velocity(case, B, fam, scale=1.0):
    """A smooth vortical field with small-scale noise on every face of a family."""
    x, y, z = _coords(B["n"], B["h"], fam)
    ph = torch.rand(6, generator=B["gen"], dtype=F64, device=DEV) * (2 * math.pi)
    k = 2 * math.pi * (1 + fam)
    a = (torch.sin(k * x + ph[0]) * torch.cos(k * y + ph[1]) * torch.cos(k * z + ph[2])
         + 0.5 * torch.cos(3 * k * x + ph[3]) * torch.sin(2 * k * y + ph[4]) * torch.cos(2 * k * z + ph[5]))
    return (a + 0.1 * _rand(B["gen"], _shape(B["n"], fam))).mul_(scale)


def _pair(a, ax, n):
    """(high, low) cells of faces 1 .. n+1 along ax."""
    return _sl(a, ax, 1, n[ax] + 2), _sl(a, ax, 0, n[ax] + 1)


def _face_mean(a, fam, n):
    """Mean of the two cells of faces 1 .. n+1 along fam; the faces beyond take the nearest cell."""
    hi, lo = _pair(a, fam, n)
    return torch.cat([_sl(a, fam, 0, 1), 0.5 * (hi + lo), _sl(a, fam, n[fam] + 1, n[fam] + 2)], dim=2 - fam)


# update_properties_by_alpha in torch
def _properties(case, B):
    n, ct, alpha = B["n"], B["ct"], B["alpha"]
    out = {}
    mixed = ct <= 1
    for key, a0, a1 in (("rho", RHO0, case["ratio"]), ("mu", MU0, MU1)):
        mix = (1.0 - alpha) * a0 + alpha * a1
        r = torch.where(mixed, mix, torch.zeros_like(mix))
        if case["spheres"]:
            todo = ct == 3
            for ax in range(3):
                for s in (1, -1):   # the low neighbour first
                    near = torch.roll(ct, s, 2 - ax) == 0
                    hit = todo & near
                    r = torch.where(hit, torch.roll(mix, s, 2 - ax), r)
                    todo = todo & ~near
        for ax in range(3):
            _sl(r, ax, 0, 1).copy_(_sl(r, ax, 1, 2))
            _sl(r, ax, n[ax] + 1, n[ax] + 2).copy_(_sl(r, ax, n[ax], n[ax] + 1))
        out[key] = r
    out["inv_rho"] = torch.where(mixed, 1.0 / out["rho"], torch.zeros_like(alpha))
    for f, name in enumerate("xyz"):
        inside = B["ft"][f] == 0
        fr = torch.where(inside, _face_mean(out["rho"], f, n), torch.ones((), dtype=F64, device=DEV))
        zero = torch.zeros_like(fr)
        out["fb" + name] = torch.where(inside, 1.0 / fr, zero)
        out["fir" + name] = out["fb" + name].clone()
        out["rho" + name] = torch.where(inside, fr, zero)
        out["mu" + name] = torch.where(inside, _face_mean(out["mu"], f, n), zero)
    return out


def _outlet(B, fb):
    """update_boundary_faces: the outlet faces (x+, mark 2) take twice the f_b of their inner neighbour."""
    if B["marks"] is not None:
        nx = B["n"][0]
        fb[0][1:-1, 1:-1, nx + 1] = 2.0 * fb[0][1:-1, 1:-1, nx]
    return fb


def _beta(B, eps, fir, fb):
    """update_poisson_beta_two_way."""
    n = B["n"]
    for f in range(3):
        w, src = fb[f], _face_mean(eps, f, n) * fir[f]
        for ax in range(3):
            hi = n[ax] + 1 + (1 if ax == f else 0)
            w, src = _sl(w, ax, 1, hi), _sl(src, ax, 1, hi)
        w.copy_(src)
    return fb


def _void(case, B):
    """Two void fractions of a settling bed (coupled cases)."""
    x, y, z = _coords(B["n"], B["h"])
    base = 0.75 + 0.2 * torch.sin(5 * x + 1.0) * torch.cos(4 * y) * torch.sin(3 * z + 0.5)
    e0 = base + 0.02 * _rand(B["gen"], _shape(B["n"]))
    return e0, e0 + 1e-4 * _rand(B["gen"], _shape(B["n"]))


def _explicit_inputs(case, seed):
    B = _base(case, seed)
    n = B["n"]
    B["dt"] = 0.1 * B["h"][0]
    B["v"] = [_velocity(case, B, f) for f in range(3)]
    B["F"] = [B["v"][f] * _face_mean(B["alpha"], f, n) * (B["dt"] / B["h"][f]) for f in range(3)]
    B["p"] = _rand(B["gen"], _shape(n))
    B["eps_old"], B["eps"] = _void(case, B) if case["coupled"] else (None, None)
    B["imp"] = [_rand(B["gen"], _shape(n, f), -1e-6, 1e-6) for f in range(3)] if case["coupled"] else None
    B["props"] = _properties(case, B)
    return B


def _solve_inputs(case, seed):
    """u*, f_b, f_inv_rho and (pressure) surface tension, void fractions, rho."""
    B = _base(case, seed)
    n = B["n"]
    B["dt"] = 1.0 if case["kind"] != "pressure" else 0.1 * B["h"][0]
    if case["fluid"] == "vof":
        P = _properties(case, B)
        fir = [P["fir" + a] for a in "xyz"]
        B["rho"] = P["rho"]
    else:
        fir = [torch.where(t == 0, 1.0, 0.0).to(F64) for t in B["ft"]]
        B["rho"] = torch.ones(_shape(n), dtype=F64, device=DEV)
    B["fir"] = fir
    fb = [a.clone() for a in fir]
    B["eps_old"], B["eps"] = _void(case, B) if case["coupled"] else (None, None)
    if case["coupled"]:
        _beta(B, B["eps"], fir, fb)
    B["fb"] = _outlet(B, fb)
    if case["kind"] == "pressure":
        vs = [_velocity(case, B, f) for f in range(3)]
        B["fs"] = []
        for f in range(3):
            hi, lo = _pair(B["alpha"], f, n)
            j = torch.zeros(_shape(n, f), dtype=F64, device=DEV)
            _sl(j, f, 1, n[f] + 2).copy_(hi - lo)
            B["fs"].append(torch.where(B["ft"][f] == 0, j * _rand(B["gen"], j.shape) * (SIGMA / B["h"][f]),
                                       torch.zeros_like(j)))
    else:
        vs = [_rand(B["gen"], _shape(n, f)) for f in range(3)]
        B["fs"] = None
    vs = [torch.where(B["ft"][f] == 0, vs[f], torch.zeros_like(vs[f])) for f in range(3)]
    if case["channel"]:
        vs[0][1:-1, 1:-1, 1] = 1.0
        vs[0][1:-1, 1:-1, n[0] + 1] = vs[0][1:-1, 1:-1, n[0]]
    B["vs"] = vs
    if case["kind"] == "adjoint":
        B["gv"] = [_rand(B["gen"], _shape(n, f)) for f in range(3)]
    return B


# ---------------------------------------------------------------------------
def _boundary():
    return BoundaryConditions(np.array(BC_TYPE, np.uint8), *(np.array(v, np.float64) for v in BC_V))


def _grid(case, B, **kw):
    n = B["n"]
    z = lambda f=None: torch.zeros(_shape(n, f), dtype=F64, device=DEV)  # noqa: E731
    a = dict(Nx_=n[0], Ny_=n[1], Nz_=n[2], dx_=B["h"][0], dy_=B["h"][1], dz_=B["h"][2], celltype_=B["ct"],
             p_=z(), p_delta_=z(), rhs_=z())
    for f, x in enumerate("xyz"):
        a[f"f_{x}type_"] = B["ft"][f]
        a[f"f_{x}bcid_"] = B["bid"][f]
        a[f"f_{x}outlet_"] = None if B["marks"] is None else B["marks"][f]
        for k in (f"f_v{x}_star_", f"f_b{x}_", f"f_inv_rho{x}_", f"f_v{x}_"):
            a[k] = z(f)
    a.update(kw)
    return DeviceGrid(**a)


def prepare(case, seed):
    kind = case["kind"]
    n = _n(case)
    if kind in ("explicit", "predict"):
        B = _explicit_inputs(case, seed)
        P = B["props"]
        kw = dict(alpha_=B["alpha"], rho_=P["rho"], rho_old_=P["rho"].clone(), mu_=P["mu"], inv_rho_=P["inv_rho"],
                  p_=B["p"], void_fraction_=B["eps"], void_fraction_old_=B["eps_old"], void_fraction_half_=B["eps"])
        mf = _mass_flux(case, B)
        for f, x in enumerate("xyz"):
            kw.update({f"f_v{x}_": B["v"][f], f"f_F{x}_accum_": B["F"][f], f"f_mf{x}_": mf[f],
                       f"f_b{x}_": P["fb" + x], f"f_inv_rho{x}_": P["fir" + x], f"f_rho{x}_": P["rho" + x],
                       f"f_mu{x}_": P["mu" + x],
                       f"f_coupling_impulse_{x}_": None if B["imp"] is None else B["imp"][f],
                       f"f_ibm_area_solid_fraction_{x}_": None if B["sf"] is None else B["sf"][f],
                       f"f_ibm_solid_fraction_{x}_": None if B["sf"] is None else B["sf"][f]})
        return {"case": case, "step": SMACStep(_grid(case, B, **kw), dt=B["dt"], g=GRAVITY, bc=_boundary())}
    B = _solve_inputs(case, seed)
    solver = B200PressureSolver(
        n, B["h"], tol=1e-8, precision=nat.PRECISION_MIXED if case["mixed"] else nat.PRECISION_FP64,
        solver_type=nat.GMG_PCG if case["channel"] else nat.PURENEUMANN_GMG_PCG)
    if kind == "adjoint":
        op = ag.StepOperator(B["alpha"], RHO0, case["ratio"], B["ct"], *B["ft"])
        return {"case": case, "solver": solver, "op": op, "dt": B["dt"], "gv": B["gv"],
                "u": [v.requires_grad_() for v in B["vs"]]}
    kw = dict(rho_=B["rho"], void_fraction_=B["eps"], void_fraction_old_=B["eps_old"])
    for f, x in enumerate("xyz"):
        kw.update({f"f_v{x}_star_": B["vs"][f], f"f_b{x}_": B["fb"][f], f"f_inv_rho{x}_": B["fir"][f],
                   f"f_s{x}_": None if B["fs"] is None else B["fs"][f]})
    g = _grid(case, B, **kw)
    step = SMACStep(g, dt=B["dt"], g=GRAVITY, bc=_boundary())
    step.pressure_solver_ = solver
    if kind == "project":
        solver.set_coefficients(g)
    return {"case": case, "step": step, "solver": solver}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "adjoint":
        u = state["u"]
        out = ag.project(u, state["solver"], state["op"], state["dt"])
        return [*(o.detach() for o in out), *torch.autograd.grad(out, u, state["gv"])]
    step = state["step"]
    g = step.grid_
    if kind == "project":
        state["solver"].project(g.f_vx_star_, g.f_vy_star_, g.f_vz_star_, step.dt_, g.p_delta_, g.f_vx_, g.f_vy_,
                                g.f_vz_)
        return [g.p_delta_, g.f_vx_, g.f_vy_, g.f_vz_]
    if kind == "pressure":
        g.p_.zero_()                # non-incremental form: p is this step's pressure
        step.solve_poisson()
        step.correct_vof_velocity()
        step.update_boundary_ghost()
        step.make_face_gradp()
        return [g.p_, g.f_vx_, g.f_vy_, g.f_vz_, g.f_gradp_x_, g.f_gradp_y_, g.f_gradp_z_, g.rhs_]
    predict = step.get_vof_vstar_rhouu_consistent_two_way if case["coupled"] else step.get_vof_vstar_rhouu_consistent
    if kind == "predict":
        predict()
        return [g.f_vx_star_, g.f_vy_star_, g.f_vz_star_]
    step.update_properties_by_alpha(RHO0, case["ratio"], MU0, MU1)
    step.compute_mass_flux_from_alpha_flux(RHO0, case["ratio"], two_way=case["coupled"])
    if case["coupled"]:
        step.update_poisson_beta_two_way()
    if case["channel"]:
        step.update_boundary_faces()
    step.calc_surface_tension(SIGMA)
    predict()
    step.update_vstar_boundary()
    out = {"rho": g.rho_, "mu": g.mu_, "inv_rho": g.inv_rho_, "kappa": g.kappa_, "gm": g.p_tmp_}
    for x in "xyz":
        out.update({"fb" + x: getattr(g, f"f_b{x}_"), "fir" + x: getattr(g, f"f_inv_rho{x}_"),
                    "frho" + x: getattr(g, f"f_rho{x}_"), "fmu" + x: getattr(g, f"f_mu{x}_"),
                    "mf" + x: getattr(g, f"f_mf{x}_"), "n" + x: getattr(g, f"n{x}_"),
                    "fs" + x: getattr(g, f"f_s{x}_"), "vs" + x: getattr(g, f"f_v{x}_star_")})
    return out


# ---------------------------------------------------------------------------
# the calls in plain torch at 64 bits
def _table(k, ids):
    t = torch.tensor(BC_TYPE if k is None else BC_V[k], dtype=U8 if k is None else F64, device=DEV)
    return t[ids.long()]


def _face_val(case, B, fam):
    """The velocity of every face of a family by the boundary rules."""
    t, v = B["ft"][fam], B["v"][fam]
    bt, bv = _table(None, B["bid"][fam]), _table(fam, B["bid"][fam])
    lam = B["sf"][fam] if B["sf"] is not None else 0.0
    zero = torch.zeros_like(v)
    wall = torch.where(bt == 2, (1.0 - lam) * bv, torch.where(bt == 4, v, zero))
    return torch.where(t == 0, v, torch.where(t == 1, wall, zero))


def _mass_flux(case, B):
    n = B["n"]
    inv_dt = 1.0 / B["dt"]
    out = []
    for f in range(3):
        q = _face_val(case, B, f)
        flux = RHO0 * q
        if case["coupled"]:
            e = _face_mean(B["eps"], f, n)
            _sl(e, f, 1, 2).copy_(_sl(B["eps"], f, 1, 2))
            _sl(e, f, n[f] + 1, n[f] + 2).copy_(_sl(B["eps"], f, n[f], n[f] + 1))
            flux = RHO0 * (e * q)
        m = flux + (case["ratio"] - RHO0) * (B["F"][f] * (B["h"][f] * inv_dt))
        if case["coupled"]:
            _sl(m, f, 0, 1).zero_()
            _sl(m, f, n[f] + 2, n[f] + 3).zero_()
        out.append(m)
    return out


def _surface_tension(case, B):
    n, h, ct, a = B["n"], B["h"], B["ct"], B["alpha"]
    zero = torch.zeros_like(a)
    inside = ct == 0

    def diff(val, ok, ax):
        hi, lo = torch.roll(val, -1, 2 - ax), torch.roll(val, 1, 2 - ax)
        okh, okl = torch.roll(ok, -1, 2 - ax), torch.roll(ok, 1, 2 - ax)
        ih, i2h = 1.0 / h[ax], 1.0 / (2.0 * h[ax])
        return torch.where(okh & okl, (hi - lo) * i2h,
                           torch.where(okh, (hi - val) * ih, torch.where(okl, (val - lo) * ih, zero)))

    g = [diff(a, inside, ax) for ax in range(3)]
    mag2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2]
    gm = torch.where(inside, torch.sqrt(mag2), zero)
    inv = torch.where(mag2 > 1e-12, 1.0 / torch.sqrt(mag2), zero)
    nrm = [torch.where(inside, c * inv, zero) for c in g]
    ok = inside & (gm > 1e-6)
    k = -(diff(nrm[0], ok, 0) + diff(nrm[1], ok, 1) + diff(nrm[2], ok, 2))
    box = torch.zeros_like(inside)
    box[1:-1, 1:-1, 1:-1] = True
    kappa = torch.where(box & (a >= 0.01) & (a <= 0.99), k, zero)
    valid = (a > 1e-2) & (a < 1 - 1e-2)
    fs = []
    for f in range(3):
        hi, lo = (lambda q: _pair(q, f, n)[0]), (lambda q: _pair(q, f, n)[1])
        kf = torch.where(hi(valid) & lo(valid), 0.5 * (hi(kappa) + lo(kappa)),
                         torch.where(hi(valid), hi(kappa), torch.where(lo(valid), lo(kappa), 0.0)))
        w = torch.where(hi(inside) & lo(inside), SIGMA * kf * (hi(a) - lo(a)) * (1.0 / h[f]), torch.zeros_like(kf))
        out = torch.zeros(_shape(n, f), dtype=F64, device=DEV)
        _sl(out, f, 1, n[f] + 2).copy_(w)
        fs.append(out)
    return nrm, kappa, gm, fs


def _minmod(p, m):
    return torch.where(p * m > 0, torch.where(p.abs() < m.abs(), p, m), torch.zeros_like(p))


def _predict(case, B, mf, fmu, mu, rho_old, inv_rho):
    """u* of the F_INTERIOR faces (0 elsewhere)."""
    n, h, dt = B["n"], B["h"], B["dt"]
    ih = [1.0 / x for x in h]
    fv = [_face_val(case, B, f) for f in range(3)]
    tw = case["coupled"]
    vol = h[0] * h[1] * h[2]
    out = []
    for A in range(3):
        lo = [1, 1, 1]
        hi = [n[0] + 1, n[1] + 1, n[2] + 1]
        lo[A] = 2

        def at(a, off=(0, 0, 0)):
            """The box's entries of an array, shifted; indices beyond the array take its edge."""
            for ax in range(3):
                i0, i1, s = lo[ax] + off[ax], hi[ax] + off[ax], a.shape[2 - ax]
                if i0 >= 0 and i1 <= s:
                    a = _sl(a, ax, i0, i1)
                else:
                    a = a.index_select(2 - ax, torch.arange(i0, i1, device=DEV).clamp_(0, s - 1))
            return a

        def e(ax, s=1, base=(0, 0, 0)):
            b = list(base)
            b[ax] += s
            return tuple(b)

        def mirrored(D, s, base=(0, 0, 0)):
            """The neighbour along D != A on side s of the face at `base`, mirrored about a wall."""
            f2 = e(D, s, base)
            inside = at(B["v"][A], base)
            ff = e(D, 1, base) if s > 0 else base
            fg = e(A, -1, ff)
            w = torch.zeros_like(inside)
            cnt = torch.zeros_like(inside)
            for q in (ff, fg):
                on = at(B["ft"][D], q) == 1
                w = w + torch.where(on, _table(A, at(B["bid"][D], q)), 0.0)
                cnt = cnt + on
            w = torch.where(cnt > 0, w / cnt.clamp(min=1.0), w)
            bt = _table(None, at(B["bid"][D], ff))
            m = torch.where((bt == 1) | (bt == 4), inside, 2.0 * w - inside)
            return torch.where(at(B["ft"][A], f2) == 0, at(B["v"][A], f2), m)

        v0 = at(B["v"][A])
        nb = {}
        for D in range(3):
            for s in (1, -1):
                nb[D, s] = at(fv[A], e(A, s)) if D == A else mirrored(D, s)
        cm = e(A, -1)
        tp, tm = at(mu) * (nb[A, 1] - v0), at(mu, cm) * (v0 - nb[A, -1])
        if tw:
            tp, tm = at(B["eps_old"]) * tp, at(B["eps_old"], cm) * tm
        tmp = 2.0 * (tp - tm) * (ih[A] * ih[A])
        for D in range(3):
            if D == A:
                continue
            sides = []
            for s in (1, -1):
                q = e(D, 1) if s > 0 else (0, 0, 0)
                qa = e(A, -1, q)
                m = 0.5 * (at(fmu[D], q) + at(fmu[D], qa))
                dv = nb[D, 1] - v0 if s > 0 else v0 - nb[D, -1]
                t = m * ((at(fv[D], q) - at(fv[D], qa)) * ih[A] + dv * ih[D])
                if tw:
                    c1 = (0, 0, 0) if s > 0 else e(D, -1)
                    c2 = e(D, 1, c1)
                    t = 0.25 * (at(B["eps_old"], c1) + at(B["eps_old"], e(A, -1, c1)) + at(B["eps_old"], c2)
                                + at(B["eps_old"], e(A, -1, c2))) * t
                sides.append(t)
            tmp = tmp + (sides[0] - sides[1]) * ih[D]
        for D in range(3):
            if D == A:
                fp = 0.5 * (at(mf[A]) + at(mf[A], e(A, 1)))
                fm = 0.5 * (at(mf[A], cm) + at(mf[A]))
            else:
                fp = 0.5 * (at(mf[D], e(A, -1, e(D, 1))) + at(mf[D], e(D, 1)))
                fm = 0.5 * (at(mf[D]) + at(mf[D], cm))
            su0 = _minmod(nb[D, 1] - v0, v0 - nb[D, -1])
            val = []
            for s, flux in ((1, fp), (-1, fm)):
                up = nb[D, s]
                far = at(fv[A], e(A, 2 * s)) if D == A else mirrored(D, s, e(D, s))
                su = _minmod(far - up, up - v0) if s > 0 else _minmod(v0 - up, up - far)
                sgn = torch.where(flux < 0, -0.5, 0.5)
                other = torch.where(at(B["ft"][A], e(D, s)) == 0, up + sgn * su, up)
                own = v0 + sgn * su0
                val.append(torch.where(flux > 0, own, other) if s > 0 else torch.where(flux > 0, other, own))
            tmp = tmp - (fp * val[0] - fm * val[1]) * ih[D]
        ir = at(inv_rho[A])
        rho_f = 0.5 * (at(rho_old) + at(rho_old, cm))
        cpl = at(B["imp"][A]) * (1.0 / vol) if B["imp"] is not None else 0.0
        dp = (at(B["p"]) - at(B["p"], cm))
        if tw:
            eo = 0.5 * (at(B["eps_old"], cm) + at(B["eps_old"]))
            en = 0.5 * (at(B["eps"], cm) + at(B["eps"]))
            tmp = tmp - eo * dp * ih[A]
            vs = (ir / en) * (eo * rho_f * v0 + dt * tmp + cpl) + dt * GRAVITY[A]
        else:
            tmp = tmp - dp * ih[A]
            vs = ir * (v0 * rho_f + cpl) + dt * (ir * tmp + GRAVITY[A])
        if B["sf"] is not None:
            vs = (1.0 - at(B["sf"][A])) * vs
        full = torch.zeros(_shape(n, A), dtype=F64, device=DEV)
        at(full).copy_(torch.where(at(B["ft"][A]) == 0, vs, 0.0))
        out.append(full)
    return out


def _exact_explicit(case, seed):
    B = _explicit_inputs(case, seed)
    P = B["props"]
    mf = _mass_flux(case, B)
    if case["kind"] == "predict":
        inv = [P["fir" + x] for x in "xyz"]
        return _predict(case, B, mf, [P["mu" + x] for x in "xyz"], P["mu"], P["rho"], inv)
    fir = [P["fir" + x] for x in "xyz"]
    fb = [P["fb" + x].clone() for x in "xyz"]
    if case["coupled"]:
        _beta(B, B["eps"], fir, fb)
    _outlet(B, fb)
    nrm, kappa, gm, fs = _surface_tension(case, B)
    vs = _predict(case, B, mf, [P["mu" + x] for x in "xyz"], P["mu"], P["rho"], fir if case["coupled"] else fb)
    nx = B["n"][0]
    if case["channel"]:
        lam = B["sf"][0] if B["sf"] is not None else torch.zeros_like(vs[0])
        vs[0][1:-1, 1:-1, 1] = (1.0 - lam[1:-1, 1:-1, 1]) * BC_V[0][2]
        vs[0][1:-1, 1:-1, nx + 1] = vs[0][1:-1, 1:-1, nx]
    out = {"rho": P["rho"], "mu": P["mu"], "inv_rho": P["inv_rho"], "kappa": kappa, "gm": gm}
    for f, x in enumerate("xyz"):
        out.update({"fb" + x: fb[f], "fir" + x: fir[f], "frho" + x: P["rho" + x], "fmu" + x: P["mu" + x],
                    "mf" + x: mf[f], "n" + x: nrm[f], "fs" + x: fs[f], "vs" + x: vs[f]})
    return out


class _Poisson:
    """The operator on the interior cells: A x = diag x - sum w x_nb, w = f_b / h^2, 0 on faces of other cells."""

    def __init__(self, case, B):
        n = B["n"]
        cell = (B["ct"] == 0)[1:-1, 1:-1, 1:-1]
        self.w, self.b = [], []
        for f in range(3):
            b = B["fb"][f]
            t = B["ft"][f]
            for ax in range(3):
                hi = n[ax] + 1 + (1 if ax == f else 0)
                b, t = _sl(b, ax, 1, hi), _sl(t, ax, 1, hi)
            b = b.clone()
            other = ~cell
            _sl(b, f, 0, n[f])[other] = 0.0
            _sl(b, f, 1, n[f] + 1)[other] = 0.0
            mid = _sl(b, f, 1, n[f])
            mid[_sl(t, f, 1, n[f]) != 0] = 0.0
            self.b.append(b)
            self.w.append(b * (1.0 / (B["h"][f] * B["h"][f])))
        self.n = n
        self.diag = sum(_sl(self.w[f], f, 0, n[f]) + _sl(self.w[f], f, 1, n[f] + 1) for f in range(3))
        self.cell = cell
        self.fluid = cell & (self.diag > 0)
        self.count = int(self.fluid.sum())
        self.inv = torch.where(self.fluid, 1.0 / torch.where(self.fluid, self.diag, 1.0), 0.0)
        self.pure = not case["channel"]

    def apply(self, x):
        y = self.diag * x
        for f in range(3):
            w = _sl(self.w[f], f, 1, self.n[f])
            _sl(y, f, 0, self.n[f] - 1).sub_(w * _sl(x, f, 1, self.n[f]))
            _sl(y, f, 1, self.n[f]).sub_(w * _sl(x, f, 0, self.n[f] - 1))
        return y

    def centre(self, x):
        x = torch.where(self.fluid, x, 0.0)
        return torch.where(self.fluid, x - x.sum() / self.count, 0.0) if self.pure else x

    def solve(self, rhs):
        """Jacobi-preconditioned CG to a relative residual of 1e-12 (None if it does not get there)."""
        b = self.centre(rhs)
        x = torch.zeros_like(b)
        r = b.clone()
        goal = 1e-24 * float((b * b).sum())
        d = None
        rz = None
        for it in range(12000):
            z = self.centre(r * self.inv)
            rz_new = (r * z).sum()
            d = z if d is None else z + (rz_new / rz) * d
            rz = rz_new
            q = self.apply(d)
            a = rz / (d * q).sum()
            x = x + a * d
            r = r - a * q
            if it % 20 == 19:
                if it % 200 == 199:
                    r = self.centre(b - self.apply(x))
                if float((r * r).sum()) <= goal:
                    return self.centre(x)
        return None


def _exact_solve(case, seed):
    B = _solve_inputs(case, seed)
    n, h, dt = B["n"], B["h"], B["dt"]
    P = _Poisson(case, B)
    ih = [1.0 / x for x in h]

    def box(a, f):
        """Faces of the cells 1..n (n + 1 along f)."""
        for ax in range(3):
            a = _sl(a, ax, 1, n[ax] + 1 + (1 if ax == f else 0))
        return a

    def div(face):
        return sum((_sl(face[f], f, 1, n[f] + 1) - _sl(face[f], f, 0, n[f])) * ih[f] for f in range(3))

    inner = lambda a: a[1:-1, 1:-1, 1:-1]  # noqa: E731
    flux = [box(B["vs"][f], f) for f in range(3)]
    extra = 0.0
    if B["eps"] is not None:
        flux = [box(_face_mean(B["eps"], f, n), f) * flux[f] for f in range(3)]
        extra = (inner(B["eps"]) - inner(B["eps_old"])) * (1.0 / dt) * (1.0 / dt)
    rhs = -div(flux) * (1.0 / dt) - extra
    if B["fs"] is not None:
        rhs = rhs - div([P.b[f] * box(B["fs"][f], f) for f in range(3)])
    rhs = torch.where(P.cell, rhs, 0.0)
    x = P.solve(rhs)
    if x is None:
        return None
    pd = torch.zeros(_shape(n), dtype=F64, device=DEV)
    inner(pd).copy_(x)

    def grad(p, f):
        out = torch.zeros(_shape(n, f), dtype=F64, device=DEV)
        hi, lo = _pair(p, f, n)
        _sl(out, f, 1, n[f] + 2).copy_((hi - lo) * ih[f])
        return out

    vel = []
    for f in range(3):
        fs = B["fs"][f] if B["fs"] is not None else 0.0
        ir = B["fir"][f]
        if case["kind"] != "pressure":          # the masked f_b of the operator
            ir = torch.zeros_like(ir)
            box(ir, f).copy_(P.b[f])
        new = B["vs"][f] + ir * dt * (fs - grad(pd, f))
        old = torch.zeros_like(new) if case["kind"] == "pressure" else B["vs"][f]
        vel.append(torch.where(B["ft"][f] == 0, new, old))
    if case["kind"] == "project":
        return [pd, *vel]
    if case["kind"] == "adjoint":
        y = []
        for f in range(3):
            w = P.b[f] * box(B["gv"][f], f)
            _sl(w, f, 0, 1).zero_()
            _sl(w, f, n[f], n[f] + 1).zero_()
            y.append(w)
        psi = P.solve(torch.where(P.fluid, div(y), 0.0))
        if psi is None:
            return None
        full = torch.zeros(_shape(n), dtype=F64, device=DEV)
        inner(full).copy_(psi)
        return [*vel, *(B["gv"][f] + grad(full, f) for f in range(3))]
    # pressure: p, ghost values, face gradients
    rho_f = torch.zeros(_shape(n), dtype=F64, device=DEV)
    inner(rho_f).copy_(rhs)
    p = pd
    src = p.clone()
    gr = torch.zeros(_shape(n), dtype=F64, device=DEV)
    idx = []
    for ax in range(3):
        i = torch.arange(n[ax] + 2, device=DEV)
        c = i.clamp(1, n[ax])
        idx.append(c)
        shp = [1, 1, 1]
        shp[2 - ax] = n[ax] + 2
        gr = gr + ((i - c).to(F64) * h[ax] * GRAVITY[ax]).reshape(shp)
    near = lambda a: a[idx[2]][:, idx[1]][:, :, idx[0]]  # noqa: E731
    p = near(src) + torch.where(B["ct"] == 2, near(B["rho"]) * gr, 0.0)
    if case["channel"]:
        vel[0][1:-1, 1:-1, n[0] + 1] = B["vs"][0][1:-1, 1:-1, n[0] + 1]     # p_delta is 0 by then
    ghost = []
    for A in range(3):
        v, D = vel[A], [ax for ax in range(3) if ax != A]
        bt, bv = _table(None, B["bid"][A]), _table(A, B["bid"][A])

        def rule(a, ax, side):
            """The ghost layer of `a`'s faces across ax, from the first two faces inside."""
            i, j = (1, 2) if side == 0 else (n[ax], n[ax] - 1)
            t, b, one, two = (_sl(q, ax, i, i + 1) for q in (bt, bv, a, a))
            two = _sl(a, ax, j, j + 1)
            return torch.where(t == 2, 2.0 * b - two, torch.where(t == 0, -two, torch.where(
                t == 4, 2.0 * one - two, torch.where(t == 1, two, one))))

        new = v.clone()
        rng = lambda a: _sl(a, A, 1, n[A] + 2)  # noqa: E731
        for k in range(2):
            G, O = D[k], D[1 - k]
            for side in (0, 1):
                dst = _sl(rng(new), G, 0 if side == 0 else n[G] + 1, 1 if side == 0 else n[G] + 2)
                _sl(dst, O, 1, n[O] + 1).copy_(_sl(rng(rule(v, G, side)), O, 1, n[O] + 1))
        for sb in (0, 1):
            for sc in (0, 1):
                b, c = D
                ib, ic = (0 if sb == 0 else n[b] + 1), (0 if sc == 0 else n[c] + 1)
                jb, jc = (1 if sb == 0 else n[b]), (1 if sc == 0 else n[c])
                pick = lambda a, i, j: _sl(_sl(rng(a), b, i, i + 1), c, j, j + 1)  # noqa: E731
                pick(new, ib, ic).copy_(0.5 * (pick(new, ib, jc) + pick(new, jb, ic)))
        ghost.append(new)
    gp = []
    for f in range(3):
        out = torch.zeros(_shape(n, f), dtype=F64, device=DEV)
        full = grad(p, f)
        w, s = out, full
        for ax in range(3):
            w, s = _sl(w, ax, 1, n[ax] + 2), _sl(s, ax, 1, n[ax] + 2)
        w.copy_(s)
        gp.append(out)
    return [p, *ghost, *gp, rho_f]


def exact(case, seed):
    if case["kind"] in ("explicit", "predict"):
        return _exact_explicit(case, seed)
    return _exact_solve(case, seed)
