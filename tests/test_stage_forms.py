"""A case's bits do not depend on how its stages are launched: with which tile size, with the next
stage's ghosts left by the stage kernel or computed by a kernel of their own, with the kernel that
also keeps the stage fields, alone or between other cases of a batch. Comparisons are exact."""
import numpy as np
import pytest

from helpers import config_for
from netflux_b200 import meshgen as mg
from netflux_b200 import solver as S
from test_reconstruction import FS, _mesh, _shuffled, _state

pytestmark = pytest.mark.gpu

FORMS = [("fp64", "Barth"), ("fp64", "NONE"), ("mixed", "Barth"), ("mixed", "NONE"), ("mixed32", "NONE")]


def _case():
    """3,024 tets (twelve tiles of 256 cells), far field at two ends, two kinds of walls."""
    m = _mesh((9, 8, 7), "all")
    return S.Mesh.from_tet_mesh(m), _state(m)


def _companion(kind):
    if kind == "128":  # flattened 50:1: tiles of 256 cells cut too many faces, tiles of 128 do not
        m = mg.box_tet_mesh(60, 6, 6, hi=(1.0, 0.02, 1.0))
    elif kind == "64":  # cells in random order: no tile but the smallest holds what its cells touch
        m = _shuffled(7, 24)
    else:  # 384,000 tets more: past the size up to which the stage kernel leaves the ghosts
        m = mg.cube_mesh(40)
    return S.Mesh.from_tet_mesh(m), _state(m)


def _run(mesh, U0, precision, n=5, **kw):
    keep = kw.pop("keep_stage_fields", False)
    cfg = config_for(precision=precision, freestream=FS, cfl=0.4, local_time_stepping=True, **kw)
    s = S.EulerSolver(cfg, mesh, U0=U0, keep_stage_fields=keep)
    s.advance(n)
    U = s.get_solver_data().get_solution()
    s.close()
    return U


@pytest.mark.parametrize("kind", ["128", "64", "ghosts"])
@pytest.mark.parametrize("precision,limiter", FORMS)
def test_alone_and_in_a_batch(precision, limiter, kind):
    mesh, U0 = _case()
    other, U1 = _companion(kind)
    alone = _run(mesh, U0, precision, limiter=limiter)
    batch = S.Mesh.concat([other, mesh])
    U = _run(batch, np.concatenate([U1, U0]), precision, limiter=limiter)
    assert np.array_equal(U[U1.shape[0]:], alone)


@pytest.mark.parametrize("kind", ["128", "64"])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed32"])
def test_first_order_alone_and_in_a_batch(precision, kind):
    mesh, U0 = _case()
    other, U1 = _companion(kind)
    alone = _run(mesh, U0, precision, spatial_order="First")
    U = _run(S.Mesh.concat([other, mesh]), np.concatenate([U1, U0]), precision, spatial_order="First")
    assert np.array_equal(U[U1.shape[0]:], alone)


@pytest.mark.parametrize("precision,limiter", FORMS)
def test_with_kept_stage_fields(precision, limiter):
    mesh, U0 = _case()
    assert np.array_equal(_run(mesh, U0, precision, limiter=limiter, keep_stage_fields=True),
                          _run(mesh, U0, precision, limiter=limiter))


@pytest.mark.parametrize("precision,limiter", FORMS)
def test_ghosts_of_the_first_stage_and_of_later_ones(precision, limiter):
    """Explicit Euler with a time step too small to move any bit: the second step's flux balance, from
    ghosts the stage kernel left, is the first one's, from the ghost kernel's."""
    mesh, U0 = _case()
    cfg = config_for(precision=precision, freestream=FS, limiter=limiter, time_scheme="ExplicitEuler")
    s = S.EulerSolver(cfg, mesh, U0=U0, keep_stage_fields=True)
    R = []
    for _ in range(3):
        s.calc_timestep(s.config)
        s.set_timestep(1e-200)
        s.step()
        R.append(s.get_solver_data().get_flux_balance())
        assert np.array_equal(s.get_solver_data().get_solution(), U0)
    s.close()
    assert np.array_equal(R[1], R[0]) and np.array_equal(R[2], R[0])
