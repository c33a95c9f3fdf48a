"""Device memory of plain-form handles.  A handle's tables and scratch bound the
largest mesh a card takes, so each form is held to what it needed when its
kernels read the metrics in the mesh's own order and kept two stage states."""
import pytest

from autoflowcfd_b200 import boxgeom, boxmesh
from autoflowcfd_b200 import ensemble as E

pytestmark = pytest.mark.gpu

# bytes per cell of these boxes with the metrics in one order and two stage states
BYTES = {
    ("bare", 1, "NONE"): 7595, ("bare", 2, "NONE"): 20394, ("bare", 3, "NONE"): 38832, ("both", 1, "NONE"): 7413,
    ("both", 2, "NONE"): 20094, ("prism", 0, "NONE"): 1474, ("prism", 1, "NONE"): 7739, ("prism", 1, "SST"): 9441,
    ("prism", 2, "NONE"): 20710, ("prism", 2, "SST"): 25834, ("prism", 3, "NONE"): 39389, ("tet", 1, "NONE"): 6903,
    ("tet", 2, "NONE"): 19320, ("tet", 3, "NONE"): 37342,
}


def handle(kind, order, turb):
    from autoflowcfd_b200.solver import B200FRSolver

    cfg = {n: {"type": "FARFIELD", "Q_free": [1.2, 60.0, 0.0, 0.0, 1e5]} for n in boxmesh.PLANE_NAMES}
    cfg["z_min"] = {"type": "WALL", "is_no_slip": True}
    sst = turb == "SST"
    parts = []
    if kind != "tet":
        parts.append(boxgeom.build_case(boxmesh.prism_box(12, 10, 9), order, cfg, wall_distance=sst))
    if kind in ("tet", "both"):
        parts.append(boxgeom.build_case(boxmesh.tet_box(5, 5, 5), order, None))
        parts[-1]["n_prism"] = parts[-1]["n_cells"]  # concatenate() joins one cell type
    case = E.concatenate(parts) if len(parts) > 1 else parts[0]
    case["n_prism"] = 0 if kind == "tet" else 12 * 10 * 9 * 2
    if kind == "bare":  # prisms without force tables
        del case["cd_wall_face"]
    return B200FRSolver(case, turb_model_name=turb)


@pytest.mark.parametrize("kind,order,turb", sorted(BYTES))
def test_plain_handle_holds_no_more_than_the_tables_in_one_order(kind, order, turb):
    s = handle(kind, order, turb)
    per_cell = s.device_bytes() / s.n_cells
    s.cleanup()
    assert per_cell <= BYTES[kind, order, turb]
