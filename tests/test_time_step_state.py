"""Which state the time step of the next step belongs to.

Comparisons are exact: the same kernels on the same bits."""
import numpy as np
import pytest

from helpers import config_for
from netflux_b200 import meshgen as mg
from netflux_b200 import solver as S

pytestmark = pytest.mark.gpu


def _batch():
    cases = [(mg.bump_mesh(8, 4, 4, h=0.05), mg.bump_freestream(0.4)),
             (mg.bump_mesh(10, 5, 5, h=0.12), mg.bump_freestream(0.6))]
    meshes = [S.Mesh.from_tet_mesh(m) for m, _ in cases]
    states = [list(fs) for (_, fs), mm in zip(cases, meshes) for _ in mm.patches()]
    U0 = np.concatenate([mg.uniform_state(mm.n_cells, fs) for (_, fs), mm in zip(cases, meshes)])
    return S.Mesh.concat(meshes), states, U0, cases[0][1]


@pytest.mark.parametrize("precision,kw", [("fp64", {}), ("fp64", dict(spatial_order="First")),
                                          ("fp64", dict(spatial_order="First", time_scheme="ExplicitEuler")),
                                          ("mixed", {}), ("mixed", dict(time_scheme="ExplicitEuler")),
                                          ("mixed32", dict(limiter="NONE"))])
def test_steps_after_a_steady_solve_move_every_case(precision, kw):
    """A case that converged early was held (its dt 0) while the others went on. The steps after the
    solve go on from its state in every case, exactly as a solver that is given that state."""
    batch, states, U0, fs = _batch()
    cfg = config_for(precision=precision, local_time_stepping=True, freestream=fs, cfl=0.4, **kw)
    a = S.EulerSolver(cfg, batch, U0=U0, patch_states=states)
    out = a.solve_steady_to(np.array([1e30, 0.0]), max_steps=41, check_every=10)  # the first case at once, the second never
    assert out["steps"][0] == 1 and not out["converged"][1]
    b = S.EulerSolver(cfg, batch, U0=a.get_solver_data().get_solution(), patch_states=states)
    dt = []
    for s in (a, b):
        s.calc_timestep(s.config)
        dt.append(s.get_solver_data().get_local_dt())
    assert (dt[0] > 0).all()
    assert np.array_equal(dt[0], dt[1])
    for n in (1, 40):
        for s in (a, b):
            s.advance(n)
        assert np.array_equal(a.get_solver_data().get_solution(), b.get_solver_data().get_solution()), n
    a.close()
    b.close()
