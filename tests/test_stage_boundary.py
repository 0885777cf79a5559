"""The boundary faces and ghosts of the stage kernel, which a warp does for its own 32 cells: chains of
hexes one wide, where a warp has more faces than lanes, and a block of them, where some warps have none.

Tolerances are the parity bars of the forms after one step against the reference-order form: 1e-12
(FP64) and 1e-5 (FP32 face work).
"""
import numpy as np
import pytest

from helpers import config_for, rel_linf
from netflux_b200 import meshgen as mg
from netflux_b200 import solver as S

pytestmark = pytest.mark.gpu
FS = (1.0, 0.4, 0.1, -0.2, 1.0 / 1.4)


@pytest.mark.parametrize("n", [(3, 1, 1), (45, 1, 1), (16, 2, 1), (12, 12, 12)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5), ("mixed32", 1e-5)])
def test_boundary_faces_by_warp(n, precision, tol):
    m = mg.box_tet_mesh(*n, jitter=0.1, seed=9, side_patches={"imin": "a", "imax": "a", "jmin": "b", "jmax": "b",
                                                              "kmin": "c", "kmax": "c"},
                        patch_types={"a": mg.FAR_FIELD, "b": mg.SLIP_WALL, "c": mg.NO_SLIP_WALL})
    rng = np.random.default_rng(4)
    V = np.tile(np.asarray(FS), (m.n_cells, 1)) + 0.03 * rng.uniform(-1, 1, (m.n_cells, 5))
    U0 = mg.prim_to_cons(V)
    mesh = S.Mesh.from_tet_mesh(m)
    for limiter in ("NONE", "Barth"):
        out = {}
        for prec in ("fp64_ref", precision):
            s = S.EulerSolver(config_for(precision=prec, freestream=FS, cfl=0.4, limiter=limiter), mesh, U0=U0)
            s.advance(1)
            out[prec] = s.get_solver_data().get_solution()
            s.close()
        assert rel_linf(out[precision], out["fp64_ref"]) <= tol, limiter
