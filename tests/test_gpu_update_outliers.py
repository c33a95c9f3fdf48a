"""The update kernels' outlier test decides per cell with warp-wide votes; at P1
four cells share a warp, so one cell's non-finite or extreme column must neither
stall its neighbours nor change them (core/fr_operators/troubled_cell.py:346-408)."""
import numpy as np
import pytest

from autoflowcfd_b200 import ensemble as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("planted", [np.inf, -np.inf, np.nan, 1e200])
def test_one_cells_extreme_value_stays_with_its_neighbours(precision, order, planted):
    from autoflowcfd_b200.solver import B200FRSolver

    spec = E.EnsembleCase((4, 3, 3), order, 0.2, 0.05, 11, (2.0, 1.0, 1.0))
    case = E.build_case(spec)
    N, S = int(case["n_cells"]), int(case["n_sps"])
    rng = np.random.default_rng(5)
    U = E.uniform_state(spec, N, S) * (1.0 + 1e-3 * rng.standard_normal((N, S, 5)))
    victim = 9
    near = {victim}
    inside = ~case["is_boundary"].astype(bool)
    for a, b in zip(case["owner_cell"][inside], case["neighbor_cell"][inside]):
        if victim in (a, b):
            near |= {int(a), int(b)}
    out = []
    for x in (None, planted):
        V = U.copy()
        if x is not None:
            V[victim, S // 3, 4] = x
        s = B200FRSolver(case, mu_molecular=E.MU, rho_inf=E.RHO_INF, vel_inf=spec.velocity, p_inf=E.P_INF,
                         precision=precision)
        s.set_state_from_cpu(V)
        out.append(s.compute_inviscid_residual().cpu().numpy())  # reports no state of its own: any error is a failure
        s.cleanup()
    clean, bad = out
    assert np.all(np.isfinite(clean))
    far = [c for c in range(N) if c not in near]
    assert np.array_equal(bad[far], clean[far])
    assert np.any(bad[victim] != clean[victim])
    if planted == 1e200 and precision == "fp64":  # a finite value: finite terms, cleared where the rule says so
        assert np.all(np.isfinite(bad))


@pytest.mark.parametrize("order", [1, 2])
def test_fp64_cell_with_a_value_beyond_fp32_at_its_middle_point(order):
    """The FP64 prism kernels subtract a reference state rounded to FP32, taken at
    the cell's middle point: a finite FP64 value that FP32 cannot hold there gives
    the residual of any other finite value, not NaN."""
    from autoflowcfd_b200.solver import B200FRSolver
    from oracle import fr_oracle as O

    spec = E.EnsembleCase((4, 3, 3), order, 0.2, 0.05, 11, (2.0, 1.0, 1.0))
    case = E.build_case(spec)
    N, S = int(case["n_cells"]), int(case["n_sps"])
    U = E.uniform_state(spec, N, S) * (1.0 + 1e-3 * np.random.default_rng(5).standard_normal((N, S, 5)))
    victim = 9
    U[victim, S // 2, 4] = 1e60
    tab = case["src_mat_table"]
    dense = {k: tab[case[k + "_index"]] for k in ("nb_src0_mat", "nb_src1_mat", "ow_src0_mat", "ow_src1_mat")}
    ref = O.inviscid_residual(O.Mesh.from_case({**case, **dense}), U)
    s = B200FRSolver(case, mu_molecular=E.MU, rho_inf=E.RHO_INF, vel_inf=spec.velocity, p_inf=E.P_INF)
    s.set_state_from_cpu(U)
    got = s.compute_inviscid_residual().cpu().numpy()
    s.cleanup()
    assert np.all(np.isfinite(ref)) and np.all(np.isfinite(got))
    # sizes of the terms that the planted pressure makes (sound speed 1e30).  The
    # outlier rule clears them; what stays is what rounding-size entries of the
    # extrapolation rows (up to 2e-15 at P2, left out on the device) make of the
    # pressure: 2e-15 of it, with a sound speed of 5e-8 of the largest, times the
    # lifting and 1 / det, below 1e3.  A value cleared on one side only is off by 1.
    scale = np.array([1e30, 1e60, 1e60, 1e60, 1e90])
    assert np.all(np.abs(got[victim] - ref[victim]).max(axis=0) <= 1e-4 * scale)
