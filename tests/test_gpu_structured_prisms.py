"""Prisms with tensor-product operators (line, plane and Kronecker factors found
at create) against the oracle and against the generic kernels.

The generic kernels take the same case once one operator entry leaves the
structure by more than the accepted 1e-12 of its operator's largest entry: 1e-10
on one c2f entry, which moves results by about that much of the flux.  Box sizes
leave 1 to 7 cells in the last warps and CTAs of the kernels (2, 3, 6 or 8 cells
per warp)."""
import numpy as np
import pytest

from autoflowcfd_b200 import boxgeom, boxmesh
from fields import per_field, scalar, worst
from oracle import fr_oracle as O

pytestmark = pytest.mark.gpu

RHO, P = 1.225, 101325.0
SHAPES = [(2, 2, 2), (3, 3, 2), (5, 3, 3), (3, 3, 3)]


def make(kind, shape, order, wall_distance=False):
    u = 60.0
    cfg = {n: {"type": "FARFIELD", "Q_free": [RHO, u, 0.0, 0.0, P]} for n in boxmesh.PLANE_NAMES}
    cfg["z_min"] = {"type": "WALL", "is_no_slip": True}
    cfg["z_max"] = {"type": "SYMMETRY"}
    cfg["y_min"] = {"type": "WALL", "is_no_slip": False}
    cfg["x_min"] = {"type": "INLET", "Q_inlet": [RHO, u, 0.0, 0.0, P]}
    cfg["x_max"] = {"type": "OUTLET", "p_outlet": P}
    if kind == "prism":
        box = boxmesh.prism_box(*shape, (0.4, 0.3, 0.2), jitter=0.1, seed=3)
    else:
        box = boxmesh.tet_box(*shape, (0.4, 0.3, 0.2), jitter=0.05, seed=3, periodic=True)
    case = boxgeom.build_case(box, order, cfg if kind == "prism" else None, wall_distance=wall_distance,
                              want_sps_coords=True)
    x = case.pop("sps_coords")
    rng = np.random.default_rng(17)
    s = lambda a: np.sin((x * a).sum(-1) * 9.0 + rng.uniform(0, 6))  # noqa: E731
    rho = RHO * (1 + 0.02 * s([1, 2, 0]))
    vel = np.stack([u * (1 + 0.1 * s([1, 0, 2])), 8 * s([0, 1, 1]), 6 * s([2, 1, 0])], -1)
    p = P * (1 + 0.004 * s([1, 1, 1]))
    U = np.concatenate([rho[..., None], rho[..., None] * vel,
                        (p / 0.4 + 0.5 * rho * (vel**2).sum(-1))[..., None]], -1)
    nut = 1e-3 * (1 + 0.3 * s([1, 0, 1]))
    return case, U, nut


def solver(case, U, precision):
    from autoflowcfd_b200.solver import B200FRSolver

    s = B200FRSolver(case, mu_molecular=2e-3, rho_inf=RHO, vel_inf=60.0, p_inf=P, precision=precision)
    s.set_state_from_cpu(U)
    return s


def evaluate(case, U, nut, precision):
    import torch

    s = solver(case, U, precision)
    out = [s.compute_inviscid_residual().cpu().numpy(),
           s.compute_viscous_residual(mu_t_field=torch.from_numpy(nut).cuda()).cpu().numpy()]
    norm = s.step()
    out += [s.U.cpu().numpy(), norm]
    s.cleanup()
    return out


def dense(case):
    c = dict(case)
    tab = c.pop("src_mat_table")
    for k in ("nb_src0_mat", "nb_src1_mat", "ow_src0_mat", "ow_src1_mat"):
        c[k] = tab[c.pop(k + "_index")]
    return O.Mesh.from_case(c)


def oracle(case, U, nut):
    m = dense(case)
    return O.inviscid_residual(m, U), O.viscous_residual(m, U, 2e-3, np.maximum(U[..., 0], 1e-10) * nut)


def rel(a, b):
    """Worst field error: mass, momentum (over the vector), energy."""
    worst = 0.0
    for sl in (slice(0, 1), slice(1, 4), slice(4, 5)):
        scale = np.abs(b[..., sl]).max()
        if scale > 0:
            worst = max(worst, float(np.abs(a[..., sl] - b[..., sl]).max() / scale))
    return worst


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("order", [1, 2])
def test_structured_prisms_against_oracle_and_generic_kernels(order, shape):
    case, U, nut = make("prism", shape, order)
    ri, rv = oracle(case, U, nut)
    broken = dict(case)
    broken["c2f_prism"] = case["c2f_prism"].copy()
    broken["c2f_prism"].flat[5] += 1e-10 * np.abs(case["c2f_prism"]).max()
    f64, g64 = evaluate(case, U, nut, "fp64"), evaluate(broken, U, nut, "fp64")
    # c2f does not enter the viscous terms: other bits there mean other kernels
    assert np.any(f64[1] != g64[1])
    assert rel(f64[0], ri) < 1e-11 and rel(f64[1], rv) < 1e-11
    # 1e-10 of an entry, times pressure over its variation (250) and the row sums
    assert rel(f64[0], g64[0]) < 1e-6 and rel(f64[1], g64[1]) < 1e-11
    assert rel(f64[2], g64[2]) < 1e-9 and abs(f64[3] - g64[3]) <= 1e-6 * g64[3]
    # FP32 operators and fluxes on deviations of a few per cent: 6e-8 times the
    # cancellation of the divergence, below 1e-4; the BF16 pairs' 2^-16 sixteen times more
    mx, gx = evaluate(case, U, nut, "mixed"), evaluate(broken, U, nut, "mixed")
    assert np.any(mx[1] != gx[1])
    assert rel(mx[0], ri) < 1e-4 and rel(mx[1], rv) < 1e-4
    assert rel(gx[0], ri) < 2e-3 and rel(gx[1], rv) < 2e-2
    assert rel(mx[2], f64[2]) < 1e-6


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [1, 2])
def test_noise_that_adds_up_in_the_folded_operator_leaves_the_structure(order, precision):
    """f2c entries off by 1.2e-13 of its largest, signed so that the row's products
    with D_fine add up: the folded W, which the kernels apply, is off by 1.6e-12 (P1)
    and 2e-11 (P2) of that row's l1 norm, over both forms' limits.  Viscous
    residuals do not see f2c: their bits tell the kernels apart."""
    case, U, nut = make("prism", (2, 2, 2), order)
    f2c, D = case["f2c_prism"], case["Dfine_prism"].reshape(case["Dfine_prism"].shape[0], -1)
    v = np.random.default_rng(0).choice([-1.0, 1.0], f2c.shape[1])
    for _ in range(50):
        v = np.sign(D @ np.sign(v @ D))
    noise = 1.2e-13 * np.abs(f2c).max() * v
    assert np.abs(noise @ D).sum() > 1.5e-12 * np.abs(f2c[0] @ D).sum()
    noisy = dict(case)
    noisy["f2c_prism"] = f2c.copy()
    noisy["f2c_prism"][0] += noise
    good, other = evaluate(case, U, nut, precision), evaluate(noisy, U, nut, precision)
    assert np.any(good[1] != other[1])
    assert rel(good[1], other[1]) < (1e-11 if precision == "fp64" else 2e-2)


def test_viscous_tets_against_oracle():
    """The generic cell kernel's viscous tiles and the staged P1 faces on tets."""
    case, U, nut = make("tet", (3, 3, 3), 1)
    ri, rv = oracle(case, U, nut)
    out = evaluate(case, U, nut, "fp64")
    assert rel(out[0], ri) < 1e-10 and rel(out[1], rv) < 1e-10


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("order", [1, 2])
def test_structured_sst_kernels_at_tile_edges(order, shape):
    """The mixed form's SST kernels of structured prisms (four P1 cells or one P2
    cell per warp) against the plain form's, which run the generic ones: one update
    of the same fields.  Operators 2e-15 apart, twice differentiated: 1e-12 of the
    fields; the sources, which differences of them make, 1e-9."""
    import torch

    from autoflowcfd_b200.solver import B200FRSolver

    case, U, nut = make("prism", shape, order, wall_distance=True)
    k = 0.5 * nut / nut.mean()
    w = k / nut
    U = np.concatenate([U, (U[..., 0] * k)[..., None], (U[..., 0] * w)[..., None]], -1)
    out = []
    for precision in ("fp64", "mixed"):
        s = B200FRSolver(case, turb_model_name="SST", mu_molecular=2e-3, rho_inf=RHO, vel_inf=60.0, p_inf=P,
                         precision=precision)
        s.set_state_from_cpu(U)
        s.set_turbulence(k, w, nut)
        dt = torch.full(k.shape, 1e-6, dtype=torch.float64, device="cuda")
        diag = [d.cpu().numpy() for d in s.compute_turbulence_source(dt, diag=True)]
        out.append(([a.cpu().numpy() for a in (s.k, s.omega, s.nu_t)], diag))
        s.cleanup()
    (f64, d64), (fmx, dmx) = out
    assert np.any(f64[0] != k) and np.any(f64[1] != w)  # the update moved them
    assert all(scalar(a, b)[1] < 1e-12 for a, b in zip(fmx, f64))
    assert all(scalar(a, b)[1] < 1e-9 for a, b in zip(dmx, d64))


@pytest.mark.parametrize("order", [0, 1, 2, 3])
def test_dual_time_stage_at_tile_edges(order):
    """Pseudo-time stages with the positivity and filter in the same kernel (eight
    cells per warp up to P1, three above): 100 cells leave remainders of both.  Two
    physical steps (BDF1, BDF2) against the oracle."""
    from autoflowcfd_b200.solver import B200FRSolver

    case, U, _ = make("prism", (5, 5, 2), order)
    ref = O.Solver(dense(case), U.copy(), 2e-3, time_scheme="dual_time", dt_step=1e-4, dual_time_inner_iter=2)
    s = B200FRSolver(case, mu_molecular=2e-3, rho_inf=RHO, vel_inf=60.0, p_inf=P, time_scheme="dual_time",
                     dual_time_inner_iter=2)
    s.set_state_from_cpu(U)
    for _ in range(2):
        n_ref, n = ref.step(), s.step(1e-4)
        assert worst(per_field(s.U, ref.U)) < 1e-12
        assert abs(n - n_ref) <= 1e-9 * n_ref
    assert worst(per_field(ref.U, U)) > 1e-9  # the steps moved the state
    s.cleanup()
