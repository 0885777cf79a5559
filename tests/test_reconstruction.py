"""The fast forms' geometry-free reconstruction against the reference-order form, which computes
gradients from the face normals: cells with listed and unlisted boundary faces (no marker lists
them, so they are dropped), one hex to several, ragged sizes around a tile of 128 or 256 cells.

Tolerances are the parity bars of the forms after one step: 1e-12 (FP64, 610 or fewer operations
of relative error 2^-53 a value, amplified by the limiter's differences) and 1e-5 (FP32 face work).
"""
import numpy as np
import pytest

from helpers import config_for, rel_linf
from netflux_b200 import meshgen as mg
from netflux_b200 import solver as S

pytestmark = pytest.mark.gpu
FS = (1.0, 0.4, 0.1, -0.2, 1.0 / 1.4)


def _mesh(n, listed):
    """n hexes of six tets; listed: "all" boundary faces, "none", or "some" (the x ends only)."""
    m = mg.box_tet_mesh(*n, jitter=0.15, seed=7, side_patches={"imin": "a", "imax": "b", "jmin": "c", "jmax": "c",
                                                               "kmin": "d", "kmax": "d"},
                        patch_types={"a": mg.FAR_FIELD, "b": mg.FAR_FIELD, "c": mg.SLIP_WALL, "d": mg.NO_SLIP_WALL})
    keep = {"all": "abcd", "some": "ab", "none": ""}[listed]
    return mg.TetMesh(m.nodes, m.tets, [x for x in m.markers if x[0] in keep],
                      {k: v for k, v in m.patch_types.items() if k in keep}, m.shape)


def _state(m, seed=3):
    rng = np.random.default_rng(seed)
    x = m.centroids()
    V = np.tile(np.asarray(FS), (m.n_cells, 1))
    for k in range(5):
        V[:, k] += 0.05 * np.sin(x @ rng.uniform(-6, 6, 3) + k) + 0.02 * rng.uniform(-1, 1, m.n_cells)
    return mg.prim_to_cons(V)


@pytest.mark.parametrize("listed", ["all", "some", "none"])
@pytest.mark.parametrize("n", [(1, 1, 1), (7, 3, 1), (4, 4, 4), (11, 4, 4), (13, 9, 5)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5), ("mixed32", 1e-5)])
def test_one_step_against_reference_order(n, listed, precision, tol):
    m = _mesh(n, listed)
    U0 = _state(m)
    mesh = S.Mesh.from_tet_mesh(m)
    for kw in (dict(limiter="Barth"), dict(limiter="NONE"), dict(limiter="Barth", local_time_stepping=True),
               dict(spatial_order="First"), dict(limiter="Barth", time_scheme="ExplicitEuler")):
        out = {}
        for prec in ("fp64_ref", precision):
            s = S.EulerSolver(config_for(precision=prec, freestream=FS, cfl=0.4, **kw), mesh, U0=U0)
            s.advance(1)
            out[prec] = s.get_solver_data().get_solution()
            s.close()
        assert rel_linf(out[precision], out["fp64_ref"]) <= tol, kw


def _shuffled(n_hex, n_bits_lost):
    """A box of n_hex^3 hexes whose cells come in random order and share one key of the renumbering
    (a far hex stretches the bounding box), so tiles hold cells from all over the mesh."""
    m = mg.box_tet_mesh(n_hex, n_hex, n_hex, jitter=0.1, seed=5)
    far = mg.box_tet_mesh(1, 1, 1, lo=(2.0 ** n_bits_lost,) * 3, hi=(2.0 ** n_bits_lost * 1.5,) * 3)
    rng = np.random.default_rng(11)
    tets = np.concatenate([m.tets, far.tets + m.nodes.shape[0]])
    tris = np.concatenate([m.markers[0][1], far.markers[0][1] + m.nodes.shape[0]])
    return mg.TetMesh(np.concatenate([m.nodes, far.nodes]), tets[rng.permutation(tets.shape[0])],
                      [("farfield", tris)], {"farfield": mg.FAR_FIELD})


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5), ("mixed32", 1e-5)])
@pytest.mark.parametrize("n_hex", [3, 7])
def test_badly_ordered_mesh(n_hex, precision, tol):
    """Cells without locality: most faces leave their tile, whose lists are the longest they can be
    (the smallest tile size takes them)."""
    m = _shuffled(n_hex, 24)
    U0 = _state(m)
    mesh = S.Mesh.from_tet_mesh(m)
    out = {}
    for prec in ("fp64_ref", precision):
        s = S.EulerSolver(config_for(precision=prec, freestream=FS, cfl=0.4, local_time_stepping=True), mesh, U0=U0)
        s.advance(2)
        out[prec] = s.get_solver_data().get_solution()
        s.close()
    assert rel_linf(out[precision], out["fp64_ref"]) <= tol


def test_separate_ghost_kernel_and_the_stage_kernels_ghosts_agree():
    """advance() with the ghosts left by the stage kernel, against nf_stage with a halo unpack before
    every stage (which has the ghost kernel compute them): the same bits."""
    import ctypes as C

    import torch

    from netflux_b200 import _lib as L
    m = _mesh((6, 4, 4), "all")
    mesh = S.Mesh.from_tet_mesh(m)
    U0 = _state(m)
    out = []
    for unpack in (False, True):
        s = S.EulerSolver(config_for(precision="fp64", freestream=FS, cfl=0.4, local_time_stepping=True), mesh, U0=U0)
        for _ in range(3):
            s.calc_timestep(s.config)
            for k in range(3):
                if unpack:  # one cell's rows back into their own place
                    cell = torch.zeros(1, dtype=torch.int64, device="cuda")
                    buf = torch.zeros(10, dtype=torch.float64, device="cuda")
                    p, b = C.cast(cell.data_ptr(), C.POINTER(C.c_int64)), C.cast(buf.data_ptr(), C.POINTER(C.c_double))
                    assert L.load().nf_halo_pack(s._h, p, 1, b) == L.NF_OK
                    assert L.load().nf_halo_unpack(s._h, p, 1, b) == L.NF_OK
                assert L.load().nf_stage(s._h, k) == L.NF_OK
        out.append(s.get_solver_data().get_solution())
        s.close()
    assert np.array_equal(out[0], out[1])


def test_kept_fields_on_unlisted_faces():
    """The gradient and limiter fields of the FP64 form, with faces missing, against the reference order."""
    m = _mesh((5, 4, 3), "some")
    U0 = _state(m)
    mesh = S.Mesh.from_tet_mesh(m)
    out = {}
    for prec in ("fp64_ref", "fp64"):
        s = S.EulerSolver(config_for(precision=prec, freestream=FS, cfl=0.4), mesh, U0=U0, keep_stage_fields=True)
        s.advance(1)
        d = s.get_solver_data()
        out[prec] = (d.get_primvars_gradient(), d.get_primvars_limiter(), d.get_flux_balance())
        s.close()
    for a, b, tol in zip(out["fp64"], out["fp64_ref"], (1e-11, 1e-10, 1e-11)):
        assert rel_linf(a, b) <= tol
