"""One handle with prisms and tetrahedra (two disjoint boxes): both cell types'
kernels run over one set of arrays, the structured prisms' in lane order and the
tets' in the mesh's, and a face record's cells are numbered across both."""
import numpy as np
import pytest

from autoflowcfd_b200 import boxgeom, boxmesh
from autoflowcfd_b200 import ensemble as E
from oracle import fr_oracle as O

pytestmark = pytest.mark.gpu

RHO, P, MU = 1.225, 101325.0, 2e-3


def make(order):
    u = 60.0
    cfg = {n: {"type": "FARFIELD", "Q_free": [RHO, u, 0.0, 0.0, P]} for n in boxmesh.PLANE_NAMES}
    cfg["z_min"] = {"type": "WALL", "is_no_slip": True}
    prisms = boxgeom.build_case(boxmesh.prism_box(4, 3, 3, (0.4, 0.3, 0.2), jitter=0.1, seed=3), order, cfg,
                                want_sps_coords=True)
    tets = boxgeom.build_case(boxmesh.tet_box(3, 3, 3, (0.4, 0.3, 0.2), jitter=0.05, seed=3, periodic=True), order,
                              None, want_sps_coords=True)
    n = int(prisms["n_cells"])
    x = np.concatenate([prisms.pop("sps_coords"), tets.pop("sps_coords")])
    tets["n_prism"] = tets["n_cells"]  # concatenate() joins one cell type; the join itself does not depend on it
    tets["cd_wall_face"] = np.zeros(tets["owner_cell"].shape, np.uint8)
    case = E.concatenate([prisms, tets])
    case["n_prism"] = n
    rng = np.random.default_rng(17)
    s = lambda a: np.sin((x * a).sum(-1) * 9.0 + rng.uniform(0, 6))  # noqa: E731
    rho = RHO * (1 + 0.02 * s([1, 2, 0]))
    vel = np.stack([u * (1 + 0.1 * s([1, 0, 2])), 8 * s([0, 1, 1]), 6 * s([2, 1, 0])], -1)
    p = P * (1 + 0.004 * s([1, 1, 1]))
    U = np.concatenate([rho[..., None], rho[..., None] * vel,
                        (p / 0.4 + 0.5 * rho * (vel**2).sum(-1))[..., None]], -1)
    return case, U, n


def rel(a, b):
    return max(float(np.abs(a[..., s] - b[..., s]).max() / max(np.abs(b[..., s]).max(), 1e-300))
               for s in (slice(0, 1), slice(1, 4), slice(4, 5)))


@pytest.mark.parametrize("order,precision", [(1, "fp64"), (2, "fp64"), (3, "fp64"), (1, "mixed")])
def test_prisms_and_tets_in_one_handle(order, precision):
    from autoflowcfd_b200.solver import B200FRSolver

    case, U, n = make(order)
    c = dict(case)
    tab = c.pop("src_mat_table")
    for k in ("nb_src0_mat", "nb_src1_mat", "ow_src0_mat", "ow_src1_mat"):
        c[k] = tab[c.pop(k + "_index")]
    m = O.Mesh.from_case(c)
    ri, rv = O.inviscid_residual(m, U), O.viscous_residual(m, U, MU, None)
    s = B200FRSolver(case, mu_molecular=MU, rho_inf=RHO, vel_inf=60.0, p_inf=P, precision=precision)
    s.set_state_from_cpu(U)
    gi, gv = s.compute_inviscid_residual().cpu().numpy(), s.compute_viscous_residual().cpu().numpy()
    cd = s.compute_aerodynamic_coefficients()
    s.step()
    assert np.all(np.isfinite(s.U.cpu().numpy()))
    s.cleanup()
    # FP64: rounding times the operators' row sums (prisms 1e3; tets 2e4, 2e11 and 2e8 at orders 1, 2 and 3, in the
    # viscous terms twice, which leaves them no digit at order 3); mixed: FP32 and BF16-pair products
    tol = {"fp64": {1: (1e-11, 1e-10), 2: (1e-11, 1e-7), 3: (1e-9, 1e-7)}, "mixed": {1: (1e-4, 2e-2)}}[precision][order]
    for part, t in ((slice(0, n), tol[0]), (slice(n, None), tol[1])):
        assert rel(gi[part], ri[part]) < t
        assert rel(gv[part], rv[part]) < t or (order == 3 and part.start == n)
    assert np.all(np.isfinite(gv))
    # the prisms' results, and the forces on their wall, are those of a handle of prisms alone
    alone = boxgeom.build_case(boxmesh.prism_box(4, 3, 3, (0.4, 0.3, 0.2), jitter=0.1, seed=3), order,
                               {**{k: {"type": "FARFIELD", "Q_free": [RHO, 60.0, 0.0, 0.0, P]} for k in boxmesh.PLANE_NAMES},
                                "z_min": {"type": "WALL", "is_no_slip": True}})
    a = B200FRSolver(alone, mu_molecular=MU, rho_inf=RHO, vel_inf=60.0, p_inf=P, precision=precision)
    a.set_state_from_cpu(U[:n])
    alone_i = a.compute_inviscid_residual().cpu().numpy()
    # P2 plain Euler faces extrapolate from the rows' nonzeros or by the full product, by the mesh's mean row: the
    # order of the sums, as against the oracle above
    assert rel(gi[:n], alone_i) < 1e-11 if (order, precision) == (2, "fp64") else np.array_equal(gi[:n], alone_i)
    assert np.array_equal(a.compute_viscous_residual().cpu().numpy(), gv[:n])
    ref = a.compute_aerodynamic_coefficients()
    a.cleanup()
    scale = max(abs(v) for v in ref.values())
    assert all(abs(cd[k] - ref[k]) <= 1e-12 * scale for k in ref)
