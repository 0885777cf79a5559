"""A case's bits do not depend on how its stages are launched: with which tile size, with the next
stage's ghosts left by the stage kernel or computed by a kernel of their own, with the kernel that
also keeps the stage fields, by kernels of one thread a cell, alone or between other cases of a
batch. Comparisons are exact."""
import ctypes as C

import numpy as np
import pytest

from helpers import config_for
from netflux_b200 import _lib as L
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
    elif kind == "order":  # cells in random order: no tile holds what its cells touch, a thread a cell
        m = _shuffled(7, 24)
    elif kind == "flat":  # 162,000 tets flattened 10:1: more than a wave of tiles, cut too often for them
        m = mg.box_tet_mesh(30, 30, 30, hi=(1.0, 0.1, 1.0))
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


def _by_cells(mesh, U0, precision, **kw):
    """Whether a step launches limiter kernels of their own (one thread a cell)."""
    cfg = config_for(precision=precision, freestream=FS, cfl=0.4, local_time_stepping=True, **kw)
    s = S.EulerSolver(cfg, mesh, U0=U0)
    ms, kms, n = C.c_double(), (C.c_double * L.NF_KERNEL_COUNT)(), (C.c_int64 * L.NF_KERNEL_COUNT)()
    assert L.load().nf_time_steps(s._h, 1, 1, C.byref(ms), kms, n) == L.NF_OK
    s.close()
    return n[L.NF_KERNEL_GRADIENT] > 0


@pytest.mark.parametrize("kind", ["128", "order", "flat", "ghosts"])
@pytest.mark.parametrize("precision,limiter", FORMS)
def test_alone_and_in_a_batch(precision, limiter, kind):
    mesh, U0 = _case()
    other, U1 = _companion(kind)
    alone = _run(mesh, U0, precision, limiter=limiter)
    assert not _by_cells(mesh, U0, precision, limiter=limiter)
    batch, Ub = S.Mesh.concat([other, mesh]), np.concatenate([U1, U0])
    assert _by_cells(batch, Ub, precision, limiter=limiter) == (kind in ("order", "flat"))
    U = _run(batch, Ub, precision, limiter=limiter)
    assert np.array_equal(U[U1.shape[0]:], alone)


@pytest.mark.parametrize("kind", ["128", "order", "flat"])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed32"])
def test_first_order_alone_and_in_a_batch(precision, kind):
    mesh, U0 = _case()
    other, U1 = _companion(kind)
    alone = _run(mesh, U0, precision, spatial_order="First")
    U = _run(S.Mesh.concat([other, mesh]), np.concatenate([U1, U0]), precision, spatial_order="First")
    assert np.array_equal(U[U1.shape[0]:], alone)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ratchet_and_converged_cases_by_cells(precision):
    """The limiter ratchet, and a case that a steady solve holds while another goes on, in a batch that
    runs by kernels of one thread a cell against each case alone."""
    mesh, U0 = _case()
    other, U1 = _companion("order")
    kw = dict(precision=precision, freestream=FS, cfl=0.3, local_time_stepping=True, limiter_ratchet_step=4)
    alone = S.EulerSolver(config_for(**kw), mesh, U0=U0)
    alone.advance(1)
    first = alone.get_solver_data().get_solution()
    alone.advance(20)
    both = S.EulerSolver(config_for(**kw), S.Mesh.concat([other, mesh, mesh]), U0=np.concatenate([U1, U0, U0]))
    out = both.solve_steady_to(np.array([0.0, 1e30, 0.0]), max_steps=21, check_every=10)
    assert list(out["steps"]) == [21, 1, 21]
    U = both.get_solver_data().get_solution()[U1.shape[0]:]
    assert np.array_equal(U[: U0.shape[0]], first)
    assert np.array_equal(U[U0.shape[0]:], alone.get_solver_data().get_solution())
    alone.close()
    both.close()


@pytest.mark.parametrize("precision,limiter", FORMS)
@pytest.mark.parametrize("kind", [None, "order"])
def test_with_kept_stage_fields(precision, limiter, kind):
    mesh, U0 = _case()
    if kind:
        other, U1 = _companion(kind)
        mesh, U0 = S.Mesh.concat([other, mesh]), np.concatenate([U1, U0])
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
