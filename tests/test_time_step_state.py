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


@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("precision,kw", [("fp64", dict(spatial_order="First")),
                                          ("fp64", dict(spatial_order="First", time_scheme="ExplicitEuler")),
                                          ("mixed", dict(time_scheme="ExplicitEuler"))])
def test_a_step_keeps_the_time_step_it_was_given(precision, kw, local):
    """FP64 first order and explicit Euler in differences: the time step of the last calc_timestep or
    set_timestep holds until the next one (Config::get_delta_time), steps between them included."""
    batch, states, U0, fs = _batch()
    rng = np.random.default_rng(3)
    U0 = U0 * (1 + 0.02 * rng.uniform(-1, 1, U0.shape))
    cfg = config_for(precision=precision, local_time_stepping=local, freestream=fs, cfl=0.4, **kw)

    def run(*calls):
        s = S.EulerSolver(cfg, batch, U0=U0, patch_states=states)
        for c in calls:
            c(s)
        out = s.get_solver_data().get_solution(), s.get_solver_data().get_local_dt() if local else None
        s.close()
        return out

    dts = []
    calc = lambda s: (s.calc_timestep(s.config), dts.append(s.config.get_delta_time()))
    step = lambda s: s.step()
    again = lambda s: s.set_timestep(dts[-1])
    once = run(calc)
    two = run(calc, step, step)
    if local:
        assert np.array_equal(two[1], once[1])  # the steps left the cells' time steps alone
    else:
        assert np.array_equal(two[0], run(calc, step, again, step)[0])
        U = run(calc, lambda s: s.set_timestep(0.5 * dts[-1]), step, step)[0]
        assert np.array_equal(U, run(calc, lambda s: s.set_timestep(0.5 * dts[-1]), step,
                                     lambda s: s.set_timestep(0.5 * dts[-1]), step)[0])


@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("time_scheme", ["TVD_RK3", "ExplicitEuler"])
def test_first_order_time_step_has_the_reference_rounding(time_scheme, local):
    """FP64 first order: however the steps are asked for, the time step has the bits of the
    reference's own operations on the primitives of the last stage's input (under explicit Euler
    those of the state before the step, so the first two time steps are the same number)."""
    batch, states, U0, fs = _batch()
    rng = np.random.default_rng(5)
    U0 = U0 * (1 + 0.02 * rng.uniform(-1, 1, U0.shape))
    cfg = config_for(precision="fp64", local_time_stepping=local, freestream=fs, cfl=0.4, spatial_order="First",
                     time_scheme=time_scheme)
    a, b, c = (S.EulerSolver(cfg, batch, U0=U0, patch_states=states) for _ in range(3))
    dts = []
    for _ in range(45):
        a.calc_timestep(a.config)
        dts.append((a.config.get_delta_time(), a.get_solver_data().get_local_dt()) if local
                   else (a.config.get_delta_time(), None))
        a.step()
    if time_scheme == "ExplicitEuler":
        assert dts[0][0] == dts[1][0]
        if local:
            assert np.array_equal(dts[0][1], dts[1][1])
    b.advance(1)
    for n in (1, 2, 36, 3, 2):  # with and without the graphs
        b.advance(n)
    c.advance(45)
    for s in (b, c):
        assert np.array_equal(s.get_solver_data().get_solution(), a.get_solver_data().get_solution())
        if local:
            assert np.array_equal(s.get_solver_data().get_local_dt(), dts[-1][1])
        assert s.advance(0) == a.advance(0)
    for s in (a, b, c):
        s.close()
