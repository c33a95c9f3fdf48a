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
        try:
            out.append(s.compute_inviscid_residual().cpu().numpy())
        except RuntimeError:
            out.append(None)
        s.cleanup()
    clean, bad = out
    assert np.all(np.isfinite(clean))
    if bad is not None:
        far = [c for c in range(N) if c not in near]
        assert np.array_equal(bad[far], clean[far])
