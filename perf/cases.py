"""Performance cases of the FR residual-and-update path, through the solver's public entry points.

Each case is a solve on a box mesh of the generator (``autoflowcfd_b200.boxgeom``) and one call that a time-marching
program repeats: a step (explicit SSP-RK3, dual time), a residual evaluation behind the solver's seam, or the replay of a
batched ensemble.  Every pass restarts from the prepared state, so passes do the same work.  ``exact`` evaluates the same
call in plain torch, in 64 bits throughout.
"""

import functools
import math

import numpy as np
import torch

from autoflowcfd_b200 import boxgeom, boxmesh
from autoflowcfd_b200 import ensemble as ens
from autoflowcfd_b200.solver import B200FRSolver

GAMMA, R_AIR, PR, PR_T, C_IP = 1.4, 287.0, 0.72, 0.9, 4.0
RHO, P_INF = 1.225, 101325.0
C_INF = math.sqrt(GAMMA * P_INF / RHO)
DT_PHYSICAL = 1e-4  # dual time: physical step


# ------------------------------------------------------------------------------------------------------------ the cases
def _case(call, flow, order, precision, nx, ny, nz, norm=False, inner=0, members=0):
    return dict(call=call, flow=flow, order=order, precision=precision, nx=nx, ny=ny, nz=nz, norm=norm, inner=inner,
                members=members)


def listed():
    c = {
        # an external-aerodynamics RANS solve (P2, SST, wall, farfield) in the production precision form, at the upper
        # end of what the serving loop admits; the step is the unit a steady solve repeats thousands of times
        "rans_mixed_p2_large": _case("step", "rans", 2, "mixed", 60, 50, 50),
        # the same solve at the lower end of the serving range, odd box: few tiles per SM, launches and tails show
        "rans_mixed_p2_small": _case("step", "rans", 2, "mixed", 25, 19, 17),
        # the plain FP64 form of the same solve (validation runs, the reference's own arithmetic)
        "rans_fp64_p2": _case("step", "rans", 2, "fp64", 24, 20, 18),
        # laminar solve with a wall bump as the serving loop runs it, mid-size, odd
        "laminar_mixed_p2": _case("step", "laminar", 2, "mixed", 59, 30, 29),
        # the same at P1, the other order that the ensemble and the serving loop draw
        "laminar_mixed_p1": _case("step", "laminar", 1, "mixed", 80, 40, 40),
        # the residual seam that an outer integrator calls: inviscid and viscous residuals one after the other
        "residual_mixed_p2": _case("residual", "laminar", 2, "mixed", 32, 16, 16),
        # smallest calls: a unit-test-sized box with the norm read every step, as solve() does
        "laminar_fp64_p1_tiny": _case("step", "laminar", 1, "fp64", 4, 3, 3, norm=True),
        # inviscid Taylor-Green on periodic P3 tets, FP64 (P3 tets have no mixed form): the residual, because the
        # operators of these tets (entries up to 6e7) leave no significant digit in the state after a whole step
        "tgv_fp64_p3_tets": _case("residual", "tgv", 3, "fp64", 16, 16, 16),
        # isentropic vortex on periodic P1 tets, the small validation configuration at its full size, norm every step
        "vortex_fp64_p1_tets": _case("step", "vortex", 1, "fp64", 16, 16, 16, norm=True),
        # order 0: the first phase of every order continuation
        "laminar_fp64_p0": _case("step", "laminar", 0, "fp64", 60, 50, 50),
        # unsteady solve: one physical step of dual time (BDF2) with a few pseudo iterations
        "dual_fp64_p2": _case("dual_time", "laminar", 2, "fp64", 20, 10, 10, inner=4),
        # batched uneven ensemble of both orders, one captured graph per step
        "ensemble_mixed": _case("ensemble", "laminar", 0, "mixed", 0, 0, 0, members=6),
    }
    return [dict(v, name=k) for k, v in c.items()]


def draw(rng):
    """One more case: a kind of the listed ones, its hex count log-uniform over that kind's range, an uneven box."""
    kind, lo, hi = rng.choice([
        (("step", "rans", 2, "mixed"), 4000, 140000), (("step", "rans", 2, "mixed"), 4000, 140000),
        (("step", "rans", 2, "fp64"), 500, 30000), (("step", "laminar", 2, "mixed"), 2000, 140000),
        (("step", "laminar", 1, "mixed"), 2000, 200000), (("step", "laminar", 1, "fp64"), 30, 60000),
        (("step", "laminar", 2, "fp64"), 500, 30000), (("residual", "laminar", 2, "mixed"), 500, 60000),
        (("residual", "laminar", 1, "mixed"), 500, 60000), (("residual", "tgv", 3, "fp64"), 30, 5000),
        (("step", "vortex", 1, "fp64"), 30, 30000), (("step", "laminar", 0, "fp64"), 2000, 200000),
        (("dual_time", "laminar", 2, "fp64"), 300, 5000), (("ensemble", "laminar", 0, "mixed"), 0, 0)])
    if kind[0] == "ensemble":
        return _case(*kind, 0, 0, 0, members=rng.randint(2, 8))
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, ay = rng.uniform(0.9, 1.6), rng.uniform(0.8, 1.2)
    s = (n / (ax * ay)) ** (1.0 / 3.0)
    nx, ny, nz = (max(3, int(f * s + 0.5)) for f in (ax, ay, 1.0))
    return _case(*kind, nx, ny, nz, norm=kind[0] == "step" and rng.random() < 0.4,
                 inner=rng.randint(2, 5) if kind[0] == "dual_time" else 0)


# ------------------------------------------------------------------------------------------------- meshes and conditions
def _conditions(flow):
    """Free-stream speed and molecular viscosity."""
    u = {"rans": 0.1, "laminar": 0.2, "tgv": 0.1, "vortex": 0.5}[flow] * C_INF
    return u, {"rans": RHO * u / 1e6, "laminar": RHO * u * 4.0 / 1e5, "tgv": 1.8e-5, "vortex": 1.8e-5}[flow]


@functools.lru_cache(maxsize=2)
def _tables(flow, order, nx, ny, nz):
    """Mesh tables of one box, its lengths and solution-point coordinates (host arrays)."""
    if flow in ("tgv", "vortex"):
        lengths = (1.0, 1.0, 1.0)
        box = boxmesh.tet_box(nx, ny, nz, lengths, jitter=0.05 if flow == "tgv" else 0.0, seed=7, periodic=True)
        case = boxgeom.build_case(box, order, None, want_sps_coords=True)
    else:
        lengths = (4.0, 2.0, 1.5)
        u = _conditions(flow)[0]
        cfg = {n: {"type": "FARFIELD", "Q_free": [RHO, u, 0.0, 0.0, P_INF]} for n in boxmesh.PLANE_NAMES}
        cfg["z_min"] = {"type": "WALL", "is_no_slip": True}
        bump = (0.06 * lengths[2], 0.4 * lengths[0], 0.5 * lengths[1], 0.25 * lengths[2]) if flow == "laminar" else None
        box = boxmesh.prism_box(nx, ny, nz, lengths, jitter=0.1, seed=2024, bump=bump)
        case = boxgeom.build_case(box, order, cfg, wall_distance=flow == "rans", want_sps_coords=True)
    return case, lengths, case.pop("sps_coords")


@functools.lru_cache(maxsize=1)
def _ensemble_tables(members):
    """Specs and tables of a small uneven ensemble: both orders, hex counts log-uniform, Mach and bump uniform."""
    specs = ens.draw_cases(members, seed=members, hex_cells=(2000, 8000))
    specs[0].order, specs[1].order = 1, 2
    return specs, [ens.build_case(s) for s in specs]


def _state(flow, lengths, xyz, seed):
    """Conserved start state at points ``xyz`` (device), made from the seed: k, omega and nu_t too for a RANS solve."""
    ph = np.random.default_rng(seed).uniform(0, 2 * math.pi, 8)
    x, y, z = (xyz[..., i] * (1.0 / lengths[i]) for i in range(3))
    sin = lambda i, a, b, c: torch.sin(2 * math.pi * (a * x + b * y + c * z) + ph[i])  # noqa: E731
    u0 = _conditions(flow)[0]
    if flow == "tgv":
        k, s = 2 * math.pi, ph / (2 * math.pi)
        xs, ys, zs = x + s[0], y + s[1], z + s[2]
        u = u0 * torch.sin(k * xs) * torch.cos(k * ys) * torch.cos(k * zs)
        v = -u0 * torch.cos(k * xs) * torch.sin(k * ys) * torch.cos(k * zs)
        w = torch.zeros_like(u)
        p = P_INF + RHO * u0**2 / 16 * (torch.cos(2 * k * xs) + torch.cos(2 * k * ys)) * (torch.cos(2 * k * zs) + 2)
        rho = p * (RHO / P_INF)
    elif flow == "vortex":
        dx, dy = (x - 0.4 - 0.2 * ph[0] / 6.3) / 0.2, (y - 0.4 - 0.2 * ph[1] / 6.3) / 0.2
        r2 = dx * dx + dy * dy
        swirl = (5.0 * C_INF / (2 * math.pi)) * torch.exp(0.5 * (1 - r2))
        th = 1 - (GAMMA - 1) * 25.0 / (8 * GAMMA * math.pi**2) * torch.exp(1 - r2)
        rho, p = RHO * th ** (1 / (GAMMA - 1)), P_INF * th ** (GAMMA / (GAMMA - 1))
        u, v, w = u0 - swirl * dy, swirl * dx, torch.zeros_like(x)
    else:
        rho = RHO * (1 + 0.01 * sin(0, 1, 1, 0) + 0.005 * sin(1, 0, 2, 1))
        u = u0 * torch.tanh(6 * z + 0.3) * (1 + 0.02 * sin(2, 1, 0, 1))
        v, w = 0.02 * u0 * sin(3, 0, 1, 1), 0.01 * u0 * sin(4, 1, 0, 1)
        p = P_INF * (1 + 0.001 * sin(5, 1, 0, 1))
    cols = [rho, rho * u, rho * v, rho * w, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v + w * w)]
    turb = ()
    if flow == "rans":  # intensity 1 %, viscosity ratio 10, both varying by a fifth
        k0 = 1.5 * (0.01 * u0) ** 2
        k = k0 * (1 + 0.2 * sin(6, 1, 1, 1))
        om = RHO * k0 / (10 * _conditions(flow)[1]) * (1 + 0.2 * sin(7, 2, 1, 0))
        cols += [rho * k, rho * om]
        turb = (k, om, k / om)
    return torch.stack(cols, -1), turb


def _solver(case, table, u, mu):
    flow = case["flow"]
    euler = flow in ("tgv", "vortex")
    return B200FRSolver(table, turb_model_name="SST" if flow == "rans" else "NONE", mu_molecular=mu, rho_inf=RHO, vel_inf=u,
                        p_inf=P_INF, inviscid_only=euler, global_dt_factor=3.0 if euler else 0.0,
                        precision=case["precision"], time_scheme="dual_time" if case["call"] == "dual_time" else "ssp_rk3",
                        dual_time_inner_iter=max(case["inner"], 1))


def _ensemble_starts(seed, specs, groups):
    """Per group of members, their perturbed free streams as one state (device)."""
    rng = np.random.default_rng(seed)
    out = []
    for members in groups:
        parts = []
        for i in members:
            n = specs[i].n_cells
            U = torch.from_numpy(ens.uniform_state(specs[i], n, _dims(specs[i].order)[0])).cuda()
            g = torch.Generator(device=U.device).manual_seed(int(rng.integers(1 << 40)))
            noise = torch.rand((n, 1, 5), generator=g, device=U.device, dtype=U.dtype) - 0.5
            scale = torch.tensor([0.01, 0.02, 0.02, 0.02, 0.002], device=U.device, dtype=U.dtype)
            ref = U.new_tensor([RHO, RHO * specs[i].velocity, RHO * specs[i].velocity, RHO * specs[i].velocity,
                                P_INF / (GAMMA - 1)])
            parts.append(U + noise * scale * ref)
        out.append(torch.cat(parts))
    return out


def prepare(case, seed):
    if case["call"] == "ensemble":
        specs, tables = _ensemble_tables(case["members"])
        e = ens.B200Ensemble(specs, precision=case["precision"], cases=tables)
        starts = _ensemble_starts(seed, specs, [g.members for g in e.groups])
        for g, s in zip(e.groups, starts):
            g.solver.U.copy_(s)
        e.capture()
        return dict(case=case, ensemble=e, starts=starts)
    table, lengths, xyz = _tables(case["flow"], case["order"], case["nx"], case["ny"], case["nz"])
    U, turb = _state(case["flow"], lengths, torch.from_numpy(xyz).cuda(), seed)
    s = _solver(case, table, *_conditions(case["flow"]))
    fields = (s.U, s.k, s.omega, s.nu_t) if turb else (s.U,)
    pairs = list(zip(fields, (U,) + turb))
    for d, src in pairs:
        d.copy_(src)
    if case["call"] == "dual_time":  # a physical level behind the state, as after a program's first step
        s.step(DT_PHYSICAL)
    return dict(case=case, solver=s, pairs=pairs)


def _by_field(U):
    out = {"density": U[..., 0], "momentum": U[..., 1:4], "energy": U[..., 4]}
    if U.shape[-1] > 5:
        out["turbulence"] = U[..., 5:]
    return out


def run(state):
    case = state["case"]
    if case["call"] == "ensemble":
        e = state["ensemble"]
        for g, start in zip(e.groups, state["starts"]):
            g.solver.U.copy_(start)
        e.replay()
        return {"p%d" % g.order: _by_field(g.solver.U) for g in e.groups}
    s = state["solver"]
    if case["call"] == "residual":
        out = {"inviscid": _by_field(s.compute_inviscid_residual())}
        if case["flow"] != "tgv":
            out["viscous"] = _by_field(s.compute_viscous_residual())
        return out
    for dst, src in state["pairs"]:  # from the start state: the same work every pass
        dst.copy_(src)
    norm = s.step(DT_PHYSICAL, want_norm=case["norm"])
    out = _by_field(s.U)
    if s.k is not None:
        out.update(k=s.k, omega=s.omega, nu_t=s.nu_t)
    if case["norm"] or case["call"] == "dual_time":
        out["norm"] = norm
    return out


# ------------------------------------------------------------------------------------------------------ work, tolerances
def _dims(order):
    return (order + 1) ** 3, (min(2 * order, 3) + 1) ** 3, (order + 1) ** 2


def _box_work(order, cells, flow, call, inner):
    """Bytes: every input (state, metrics, face normals and indices) once and every output once.  Operations: the
    operator contractions of one residual evaluation times the evaluations of the call, plus the filter."""
    S, Fn, P = _dims(order)
    faces = 4.0 * cells if flow in ("rans", "laminar") else 3.0 * cells
    nv = 7 if flow == "rans" else 5
    fields = nv + (3 if flow == "rans" else 0)
    visc = flow in ("rans", "laminar")
    metrics = 80 * S + (80 * Fn if order else 8)
    outputs = 2 * 5 * S if call == "residual" else S * fields
    by = cells * (8 * (S * fields + outputs) + metrics) + faces * (24 * P + 24)
    width = 18 if visc else 5
    one = 2 * Fn * S * 5 + 2 * S * 3 * Fn * 5 + 2 * 6 * P * S * width + (2 * 3 * S * S * 9 if visc else 0)
    one = 100 * 4 if order == 0 else one
    evals = {"step": 3, "residual": 1, "dual_time": 1 + 3 * inner}[call]
    fl = cells * (evals * (one + (0 if call == "residual" else 2 * S * S * 5)) + (2 * 3 * S * S * 14 if flow == "rans" else 0))
    return by, fl


def work(case):
    if case["call"] == "ensemble":
        specs = _ensemble_tables(case["members"])[0]
        parts = [_box_work(s.order, s.n_cells, "laminar", "step", 0) for s in specs]
    else:
        cells = case["nx"] * case["ny"] * case["nz"] * (6 if case["flow"] in ("tgv", "vortex") else 2)
        parts = [_box_work(case["order"], cells, case["flow"], case["call"], case["inner"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """About four times the error against ``exact`` (relative 2-norm, the worst output of the case)."""
    if case["call"] == "residual":
        if case["flow"] == "tgv":  # sums over operator entries up to 6e7 and weights up to 2e7: 1e-7 to 5e-6 seen
            return {"rel": 2e-5}
        # mixed form: 5e-5 seen on the inviscid outputs, 2.5e-3 on the viscous energy (conduction: a cancelling
        # divergence of temperature gradients)
        return {"rel": 1e-2}
    if case["precision"] == "mixed":  # 3.3e-8 seen on the momentum, 1e-6 on the residual norm
        return {"rel": 4e-6 if case["norm"] else 1.5e-7}
    return {"rel": 3e-14}  # 1e-16 to 8e-15 seen: FP64 sums in another order, scaled by the small time step


# ------------------------------------------------------------------------- the same calls in plain torch, 64 bits
def _prim(U):
    rho = U[..., 0].clamp(min=1e-10)
    v = U[..., 1:4] / rho[..., None]
    p = (GAMMA - 1) * rho * (U[..., 4] / rho - 0.5 * (v * v).sum(-1))
    return torch.cat([rho[..., None], v, p[..., None]], -1)


def _euler(q):
    rho, v, p = q[..., 0], q[..., 1:4], q[..., 4]
    m = rho[..., None] * v
    F = q.new_empty(q.shape[:-1] + (3, 5))
    F[..., 0] = m
    F[..., 1:4] = m[..., :, None] * v[..., None, :] + p[..., None, None] * torch.eye(3, dtype=q.dtype, device=q.device)
    F[..., 4] = (GAMMA / (GAMMA - 1) * p + 0.5 * rho * (v * v).sum(-1))[..., None] * v
    return F


def _viscous(q, gv, gT, mu, mut):
    mt = (mu + mut)[..., None, None]
    eye = torch.eye(3, dtype=q.dtype, device=q.device)
    tau = mt * (gv + gv.transpose(-1, -2)) - 2.0 / 3.0 * mt * gv.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] * eye
    cp = GAMMA * R_AIR / (GAMMA - 1)
    k = mu * cp / PR + mut * cp / PR_T
    G = torch.zeros(q.shape[:-1] + (3, 5), dtype=q.dtype, device=q.device)
    G[..., 1:4] = tau
    G[..., 4] = (tau * q[..., None, 1:4]).sum(-1) - k[..., None] * gT
    return G


def _ausm(L, R, n):
    """AUSM+up with the low-Mach correction."""
    rl, rr = L[..., 0].clamp(min=1e-6), R[..., 0].clamp(min=1e-6)
    pl, pr = L[..., 4].clamp(min=10.0), R[..., 4].clamp(min=10.0)
    ul, ur = (L[..., 1:4] * n).sum(-1), (R[..., 1:4] * n).sum(-1)
    al, ar = (GAMMA * pl / rl).clamp(min=1e-10).sqrt(), (GAMMA * pr / rr).clamp(min=1e-10).sqrt()
    ml, mr = ul / al.clamp(min=1e-10), ur / ar.clamp(min=1e-10)
    ah, rh = 0.5 * (al + ar), 0.5 * (rl + rr)
    mb = (ul * ul + ur * ur) / (2 * ah * ah)
    m0 = mb.clamp(min=0.01).clamp(max=1.0).sqrt()
    fa = (m0 * (2 - m0)).clamp(min=1e-6)

    def split(M, s):  # s = +1: M+, P+ ; -1: M-, P-
        far = M.abs() >= 1
        mach = torch.where(far, 0.5 * (M + s * M.abs()), s * 0.25 * (M + s) ** 2 + s * 0.1875 * (M * M - 1) ** 2)
        pres = torch.where(far, 0.5 * (1 + s * torch.sign(M)),
                           0.25 * ((M + s) ** 2 * (2 - s * M) + s * 0.5 * M * (M * M - 1) ** 2))
        return mach, pres

    (mp, pp), (mm, pm) = split(ml, 1.0), split(mr, -1.0)
    mpp = -(0.25 / fa) * (1 - mb).clamp(min=0.0) * (pr - pl) / (rh * ah * ah)
    md = 0.5 * (rl * al + rr * ar) * (mp + mm + mpp)
    ph = pp * pl + pm * pr - 0.75 * pp * pm * (rl + rr) * fa * ah * (ur - ul)
    hl = GAMMA / (GAMMA - 1) * pl / rl + 0.5 * (L[..., 1:4] ** 2).sum(-1)
    hr = GAMMA / (GAMMA - 1) * pr / rr + 0.5 * (R[..., 1:4] ** 2).sum(-1)
    up = md >= 0
    mom = md[..., None] * torch.where(up[..., None], L[..., 1:4], R[..., 1:4]) + ph[..., None] * n
    return torch.cat([md[..., None], mom, (md * torch.where(up, hl, hr))[..., None]], -1)


def _suppress(R, ref):
    S = R.shape[1]
    a = R.abs().sort(dim=1)[0]
    med = a[:, S // 2] if S % 2 else 0.5 * (a[:, S // 2 - 1] + a[:, S // 2])
    thr = torch.maximum(med, 1e-9 * ref.abs().mean(1)).clamp(min=1e-300)
    return torch.where(R.abs() > 1e4 * thr[:, None], torch.zeros_like(R), R)


def _positivity(U):
    rho = U[..., 0].clamp(min=1e-6)
    v = U[..., 1:4] / rho[..., None]
    vm = v.norm(dim=-1, keepdim=True)
    v = torch.where(vm > 1e4, v * (1e4 / vm), v)
    mom = torch.where(vm > 1e4, rho[..., None] * v, U[..., 1:4])
    ke = 0.5 * rho * (v * v).sum(-1)
    low = (GAMMA - 1) * (U[..., 4] - ke) < 1.0
    E = torch.where(low, 1.0 / (GAMMA - 1) + ke, U[..., 4])
    cols = [rho[..., None], mom, E[..., None]]
    if U.shape[-1] > 5:
        cols += [U[..., 5:6].clamp(min=0.0), U[..., 6:7].clamp(min=1e-8)]
    return torch.cat(cols, -1)


class _Plain:
    """The discretisation on one mesh of one cell type."""

    def __init__(self, t, mu, inviscid_only):
        dev = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(d)  # noqa: E731
        self.N, self.S, self.order, self.mu, self.inviscid_only = int(t["n_cells"]), int(t["n_sps"]), int(t["order"]), mu, inviscid_only
        kind, ct = ("prism", 0) if int(t["n_prism"]) else ("tet", 1)
        N, S = self.N, self.S
        self.det, self.inv = dev(t["det_jacs"]), dev(t["inv_jacs"]).reshape(N, S, 3, 3)
        self.adj = self.det[..., None, None] * self.inv
        self.D = dev(t["D_3d_" + kind])  # (S, S, 3): d/d(axis m) of basis j at point s
        self.filt = dev(t["filter_" + kind])
        if self.order:
            self.c2f, self.Df, self.f2c = (dev(t[k + kind]) for k in ("c2f_", "Dfine_", "f2c_"))
            self.adjf = dev(t["det_jacs_fine"])[..., None, None] * dev(t["inv_jacs_fine"]).reshape(N, -1, 3, 3)
        self.P = t["boundary_extrap"].shape[3]
        self.E = dev(t["boundary_extrap"][ct]).reshape(6 * self.P, S)
        self.gl, self.gr = dev(t["g_left"]), dev(t["g_right"])
        self.fp, self.co = (dev(t[k], torch.int64).reshape(3, S) for k in ("dist_fp_of_sp", "dist_axis_coord_of_sp"))
        self.vol, self.area = dev(t["cell_volumes"]), dev(t["true_area_weight"])
        self.normal = dev(t["true_normal"])
        i64 = {k: dev(t[k], torch.int64) for k in ("owner_cell", "neighbor_cell", "owner_axis", "neighbor_axis", "bc_group", "bc_type")}
        self.own, self.nbr, self.bcg, self.bct = i64["owner_cell"], i64["neighbor_cell"], i64["bc_group"], i64["bc_type"]
        self.axis = {"nb": i64["owner_axis"], "ow": i64["neighbor_axis"].clamp(min=0)}  # own axis of the side that reads "nb" / "ow"
        self.side = {"nb": dev(t["owner_side"]), "ow": dev(t["neighbor_side"])}
        self.bnd = dev(t["is_boundary"], torch.bool)
        prim = {"nb": dev(t["owner_is_primary"], torch.bool), "ow": dev(t["neighbor_is_primary"], torch.bool)}
        self.slots = {"nb": prim["nb"].nonzero()[:, 0], "ow": (~self.bnd & prim["ow"]).nonzero()[:, 0]}
        self.bcQ, self.bcv = dev(t["bc_Q"]), dev(t["bc_wall_vel"])
        self.mats = dev(t["src_mat_table"])
        self.src = {}
        for w in ("nb", "ow"):
            self.src[w] = [dev(t[w + k], torch.int64) for k in ("_src0_cell", "_src0_mat_index", "_src1_idx", "_src1_cell", "_src1_mat_index")]
        self.wd = dev(t["wall_distance"]) if t.get("wall_distance") is not None else None

    def grad(self, f):
        """Physical gradient of fields (N, S, n) -> (N, S, n, 3)."""
        ref = torch.stack([torch.matmul(self.D[:, :, m], f) for m in range(3)], -1)
        return torch.matmul(ref, self.inv)

    def div(self, D, F):
        """sum over points and axes of D (S, J, 3) times F (N, J, 3, n)."""
        return sum(torch.matmul(D[:, :, m], F[:, :, m]) for m in range(3))

    def own_side(self, f, faces, w, X):
        """Own cell's values at the flux points of the given face sides."""
        cell = (self.own if w == "nb" else self.nbr)[faces]
        code = self.axis[w][faces] * 2 + (self.side[w][faces] > 0)
        return X[cell, code]

    def faces_of(self, f):
        return torch.matmul(self.E, f).reshape(self.N, 6, self.P, f.shape[-1])

    def other_side(self, f, faces, w):
        """The other side's values by the mesh's interpolation matrices (zero where there is no source)."""
        c0, m0, i1, c1, m1 = self.src[w]
        out = f.new_zeros((len(faces), self.P, f.shape[-1]))
        i = i1[faces]
        for cells, mats, rows in ((c0[faces], m0[faces], c0[faces] >= 0),
                                  (c1[i.clamp(min=0)] if len(c1) else i, m1[i.clamp(min=0)] if len(c1) else i, i >= 0)):
            for m in torch.unique(mats[rows]).tolist():
                at = (rows & (mats == m)).nonzero()[:, 0]
                out[at] += torch.matmul(self.mats[m], f[cells[at]])
        return out

    def ghost(self, q, faces):
        n, code = self.normal[faces], self.bcg[faces]
        typ = self.bct[code][:, None, None]
        wall = torch.cat([q[..., :1], 2 * self.bcv[code][:, None] - q[..., 1:4], q[..., 4:]], -1)
        return torch.where(typ == 0, wall, self.bcQ[code][:, None].expand_as(q))  # no-slip wall, farfield

    def lift(self, jump, faces, w, sign, out):
        cell = (self.own if w == "nb" else self.nbr)[faces]
        ax, sd = self.axis[w][faces], self.side[w][faces]
        co, fp = self.co[ax], self.fp[ax]
        g = torch.where((sd > 0)[:, None], self.gr[co], self.gl[co])
        c = g[..., None] * torch.gather(jump, 1, fp[..., None].expand(-1, -1, jump.shape[-1]))
        out.index_add_(0, cell, sign * c / self.det[cell][..., None])

    def finite_volume(self, q):
        q, n = q[:, 0], self.normal[:, 0]
        other = q[torch.where(self.bnd, self.own, self.nbr)]
        b = self.bnd.nonzero()[:, 0]
        last = torch.full((self.N,), -1, dtype=torch.int64, device=q.device).scatter_reduce_(0, self.own[b], b, "amax")
        last = last[self.own[b]]  # one ghost state per cell: its last boundary face's
        other[b] = self.ghost(q[self.own[b]][:, None], last)[:, 0]
        F = _ausm(q[self.own], other, n) * self.area
        R = torch.zeros_like(q).index_add_(0, self.own, -F / self.vol[self.own][:, None])
        i = (~self.bnd).nonzero()[:, 0]
        return R.index_add_(0, self.nbr[i], F[i] / self.vol[self.nbr[i]][:, None])[:, None]

    def residuals(self, U, mut=None):
        """Inviscid and viscous dU/dt of the five mean-flow variables."""
        q = _prim(U)
        visc = not self.inviscid_only
        mut = torch.zeros_like(q[..., 0]) if mut is None else mut
        Ri = Rv = None
        if self.order:
            Ft = torch.matmul(self.adjf, _euler(torch.matmul(self.c2f, q)))
            Ri = -torch.matmul(self.f2c, self.div(self.Df, Ft)) / self.det[..., None]
        f = q
        if visc:
            T = q[..., 4:] / (q[..., :1] * R_AIR)
            g = self.grad(torch.cat([q[..., 1:4], T], -1))
            Rv = self.div(self.D, torch.matmul(self.adj, _viscous(q, g[:, :, :3], g[:, :, 3], self.mu, mut))) / self.det[..., None]
            f = torch.cat([q, g.reshape(self.N, self.S, 12), mut[..., None]], -1)
        X, A = self.faces_of(f), self.faces_of(self.adj.reshape(self.N, self.S, 9))
        for w, s0 in (("nb", 1.0), ("ow", -1.0)):
            fa = self.slots[w]
            if not len(fa):
                continue
            ax, sd = self.axis[w][fa], self.side[w][fa]
            own, oth = self.own_side(f, fa, w, X), self.other_side(f, fa, w)
            arow = self.own_side(None, fa, w, A).reshape(len(fa), self.P, 3, 3)[torch.arange(len(fa), device=f.device), :, ax]
            b = self.bnd[fa]
            if b.any():
                oth[b] = own[b]
                oth[b, :, :5] = self.ghost(own[b][..., :5], fa[b])
            if self.order:
                mag = arow.norm(dim=-1, keepdim=True).clamp(min=1e-300)
                d, tn = arow / mag * sd[:, None, None], s0 * self.normal[fa]
                d = torch.where(((d * tn).sum(-1) < 0.5)[..., None], tn, d)
                jump = _ausm(own[..., :5], oth[..., :5], d) * mag * sd[:, None, None]
                jump = jump - torch.matmul(arow[..., None, :], _euler(own[..., :5]))[..., 0, :]
                self.lift(jump, fa, w, -1.0, Ri)
            if visc:
                flux = lambda x: torch.matmul(arow[..., None, :], _viscous(x[..., :5], x[..., 5:14].unflatten(-1, (3, 3)), x[..., 14:17], self.mu, x[..., 17]))[..., 0, :]  # noqa: E731,E501
                jump = flux(0.5 * (own + oth)) - flux(own)
                if b.any():
                    h = self.det[self.own[fa[b]]].mean(1) ** (1.0 / 3.0)
                    eta = C_IP * (self.mu + own[b][..., 17]) / h[:, None] * arow[b].norm(dim=-1) * sd[b][:, None]
                    jump[b, :, 1:4] -= eta[..., None] * (own[b][..., 1:4] - oth[b][..., 1:4])
                self.lift(jump, fa, w, 1.0, Rv)
        if not self.order:
            Ri = self.finite_volume(q)
        Ri = _suppress(Ri, U[..., :5])
        return Ri, _suppress(Rv, U[..., :5]) if visc else torch.zeros_like(Ri)

    def rate(self, U, nut):
        Ri, Rv = self.residuals(U, None if nut is None else U[..., 0].clamp(min=1e-10) * nut)
        return torch.cat([Ri + Rv, torch.zeros_like(U[..., 5:])], -1)

    def local_dt(self, U, nut, factor):
        rho = U[..., 0].clamp(min=1e-10)
        v = U[..., 1:4] / rho[..., None]
        p = ((U[..., 4] - 0.5 * rho * (v * v).sum(-1)) * 0.4).clamp(min=1.0)
        wave = (v.norm(dim=-1) + (1.4 * p / rho).clamp(min=1e-10).sqrt()).clamp(min=1e-10)
        h = (self.vol.abs() ** (1.0 / 3.0))[:, None]
        o = 2 * self.order + 1
        mu = self.mu + rho * nut if nut is not None else self.mu * torch.ones_like(rho)
        mfs = self.adj.norm(dim=-1).sum(-1)
        dt = torch.minimum(0.1 / o * h / wave, 0.25 * 0.1 / (o * o) * rho * h * h / mu.clamp(min=1e-30))
        dt = torch.minimum(dt, 0.1 * self.det.abs() / (mfs * wave).clamp(min=1e-300))
        return factor * dt.min() * torch.ones_like(dt) if factor else dt

    def filtered(self, U):
        return torch.cat([torch.matmul(self.filt, U[..., :5]), U[..., 5:]], -1)

    def rk3(self, U0, dt, rate, L0):
        d = dt[..., None]
        U = self.filtered(_positivity(U0 + d * L0))
        U = self.filtered(_positivity(0.75 * U0 + 0.25 * U + 0.25 * d * rate(U)))
        return self.filtered(_positivity(U0 / 3 + 2.0 / 3.0 * U + 2.0 / 3.0 * d * rate(U)))

    def transport(self, phi, gamma, gphi, rho, vel, wall_zero):
        """Convection plus diffusion of one turbulence scalar, per unit density."""
        n = lambda x: x[..., None]  # noqa: E731
        Fc, Fd = n(rho * phi) * vel, n(gamma) * gphi
        both = torch.matmul(self.adj, torch.stack([Fc, Fd], -1))
        vol = self.div(self.D, both) / n(self.det)
        allf = torch.arange(len(self.own), device=phi.device)
        f = torch.cat([n(rho), vel, n(phi), n(gamma)], -1)
        own, oth = self.own_side(f, allf, "nb", self.faces_of(f)), self.other_side(f[..., 4:], allf, "nb")
        po, pn, go, gn = own[..., 4], oth[..., 0], own[..., 5], oth[..., 1]
        none = ((self.src["nb"][0] < 0) & (self.src["nb"][2] < 0))[:, None]
        wall = (self.bct[self.bcg] == 0)[:, None]
        gn = torch.where(none, go, gn)
        pn = torch.where(none, torch.where(wall, -po, po) if wall_zero else po, pn)
        m = (n(own[..., 0]) * own[..., 1:4] * self.normal).sum(-1)
        jump = torch.stack([m * (torch.where(m >= 0, po, pn) - po), 0.5 * (go + gn) * (0.5 * (po + pn) - po)], -1)
        corr = torch.zeros_like(vol)
        self.lift(jump, allf, "nb", -1.0, corr)
        self.lift(jump[~self.bnd], allf[~self.bnd], "ow", 1.0, corr)
        R = -vol[..., 0] + corr[..., 0] - vol[..., 1] - corr[..., 1]
        return _suppress(n(R / rho), n(phi))[..., 0]

    def sst(self, U, k, om, dt):
        """Source, transport and point-implicit update of k and omega; returns k, omega, nu_t."""
        b1, b2, bs, s2, a1, kap = 0.075, 0.0828, 0.09, 0.856, 0.31, 0.41
        rho = U[..., 0].clamp(min=1e-10)
        vel, d = U[..., 1:4] / rho[..., None], self.wd.clamp(min=1e-10)
        g = self.grad(torch.cat([U[..., 1:4], k[..., None], om[..., None]], -1))

        def clipped(x):
            mag = x.norm(dim=-1, keepdim=True)
            return torch.where(mag > 1e6, x * (1e6 / mag.clamp(min=1e-10)), x)

        gk, gw = clipped(g[:, :, 3]), clipped(g[:, :, 4])
        sij = 0.5 * (g[:, :, :3] + g[:, :, :3].transpose(-1, -2))
        Sm, gd = (2 * (sij * sij).sum((-1, -2))).sqrt(), (gk * gw).sum(-1)

        def blend(nu):
            kk, ww = k.clamp(min=1e-10), om.clamp(min=1e-10)
            cd = (2 * rho * s2 / ww * gd).clamp(min=1e-10)
            arg = torch.maximum(kk.sqrt() / (bs * ww * d), 500 * nu / (d * d * ww))
            return torch.tanh(torch.minimum(arg, 4 * rho * s2 * kk / (cd * d * d)).clamp(max=1e75) ** 4)

        nu = 1.8e-5 / rho
        F1 = blend(nu)
        F2 = torch.tanh(torch.maximum(2 * k.clamp(min=1e-10).sqrt() / (bs * om * d), 500 * nu / (d * d * om)).clamp(max=1e150) ** 2)
        beta = F1 * b1 + (1 - F1) * b2
        nut = a1 * k.clamp(min=1e-10) / torch.maximum(a1 * om.clamp(min=1e-10), F2 * Sm.clamp(min=1e-10))
        nut = torch.minimum(nut, 1e5 * nu)
        c1, c2 = b1 / bs - 0.5 * kap**2 / math.sqrt(bs), b2 / bs - s2 * kap**2 / math.sqrt(bs)
        Sk = torch.minimum(nut * rho * Sm * Sm, 10 * bs * rho * k * om) - rho * bs * k * om
        Sw = rho * (F1 * c1 + (1 - F1) * c2) * Sm * Sm - rho * beta * om * om + 2 * rho * (1 - F1) * s2 / om * gd
        Ft = blend(self.mu / rho)
        tk = self.transport(k, self.mu + (Ft * 0.85 + (1 - Ft)) * rho * nut, g[:, :, 3], rho, vel, True)
        tw = self.transport(om, self.mu + (Ft * 0.5 + (1 - Ft) * s2) * rho * nut, g[:, :, 4], rho, vel, False)
        kn = k + dt * (Sk / rho / (1 + dt * bs * om) + tk)
        wn = om + dt * (Sw / rho / (1 + dt * beta * om) + tw)
        return kn.clamp(min=1e-12), wn.clamp(min=1e-12), nut

    def dual_time(self, U0, dt_local, inner):
        """One physical step from a level n-1 equal to level n (BDF2), ``inner`` pseudo iterations."""
        def rate(U):
            return self.rate(U, None) - (3 * U - 3 * U0) / (2 * DT_PHYSICAL)

        U, cfl, prev, L = U0, 0.1, None, rate(U0)
        first = float(L.norm())
        for it in range(inner):
            L = rate(U)
            cur = float(L.norm())
            if cur < first * 1e-6 or (it and cur < 1e-4):
                break
            if it and cur / prev < 0.5:
                cfl = min(cfl * 1.5, 10.0)
            elif it and cur / prev > 1.0:
                cfl = max(cfl * 0.5, 0.1)
            prev = cur
            new = self.filtered(_positivity(self.rk3(U, dt_local * cfl, rate, L)))
            if float((new - U).norm()) < 1e-10:
                break
            U = new
        return U


def exact(case, seed):
    """What ``run`` returns for these inputs, in plain torch and 64 bits."""
    flow = case["flow"]
    if case["call"] == "ensemble":
        specs, tables = _ensemble_tables(case["members"])
        orders = sorted({s.order for s in specs})
        groups = [[i for i, s in enumerate(specs) if s.order == o] for o in orders]
        starts = _ensemble_starts(seed, specs, groups)
        out = {}
        for order, members, U0 in zip(orders, groups, starts):
            ends = []
            for i, U in zip(members, U0.split([specs[i].n_cells for i in members])):
                m = _Plain(tables[i], ens.MU, False)
                rate = lambda x, m=m: m.rate(x, None)  # noqa: E731
                ends.append(m.rk3(U, m.local_dt(U, None, 0.0), rate, rate(U)))
            out["p%d" % order] = _by_field(torch.cat(ends))
        return out
    table, lengths, xyz = _tables(flow, case["order"], case["nx"], case["ny"], case["nz"])
    U, turb = _state(flow, lengths, torch.from_numpy(xyz).cuda(), seed)
    m = _Plain(table, _conditions(flow)[1], flow in ("tgv", "vortex"))
    if case["call"] == "residual":
        return {k: _by_field(r) for k, r in zip(("inviscid", "viscous"), m.residuals(U)) if k == "inviscid" or flow != "tgv"}
    nut = turb[2] if turb else None
    dt = m.local_dt(U, nut, 3.0 if flow in ("tgv", "vortex") else 0.0)
    out = {}
    if turb:
        k, om, nut = m.sst(U, turb[0], turb[1], dt)
        out.update(k=k, omega=om, nu_t=nut)
    rate = lambda x: m.rate(x, nut)  # noqa: E731
    L0 = rate(U)
    if case["norm"] or case["call"] == "dual_time":
        out["norm"] = float(L0.norm()) / math.sqrt(L0.numel())
    if case["call"] == "dual_time":
        out.update(_by_field(m.dual_time(U, dt, case["inner"])))
    else:
        out.update(_by_field(m.rk3(U, dt, rate, L0)))
    return out
