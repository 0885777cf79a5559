"""The NF_DEBUG build on what the golden cases of test_debug_build.py do not reach: the form with FP32
copies with and without the limiter, first order, unlisted faces, kept stage fields, a mesh whose tiles
have 128 cells, and one that runs by kernels of one thread a cell. Valid meshes: nothing reported, the release build's bits."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_debug_build import ROOT

pytestmark = pytest.mark.gpu

RUNS = r"""
import sys
import numpy as np
from helpers import config_for
from netflux_b200 import _lib as L, meshgen as mg, solver as S
from test_reconstruction import FS, _mesh, _shuffled, _state


def runs():
    meshes = dict(listed=_mesh((9, 8, 7), "all"), some=_mesh((7, 5, 3), "some"), order=_shuffled(7, 24),
                  flat=mg.box_tet_mesh(60, 6, 6, hi=(1.0, 0.02, 1.0)))
    for name, m in meshes.items():
        mesh, U0 = S.Mesh.from_tet_mesh(m), _state(m)
        for prec in ("fp64", "mixed", "mixed32"):
            for kw in (dict(limiter="Barth"), dict(limiter="NONE"), dict(spatial_order="First")):
                for keep in (False, True):
                    s = S.EulerSolver(config_for(precision=prec, freestream=FS, cfl=0.3, local_time_stepping=True, **kw),
                                      mesh, U0=U0, keep_stage_fields=keep)
                    s.advance(3)
                    s.synchronize()
                    yield "_".join([name, prec, *map(str, kw.values()), str(keep)]), s.get_solver_data().get_solution()
                    s.close()
"""
CHILD = r"""
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
{runs}
assert L.LIB_PATH.endswith("libnetflux_b200_debug.so"), L.LIB_PATH
for name, U in runs():
    np.save({tmp!r} + "/" + name + ".npy", U)
print("debug ok")
"""


def test_debug_build_on_every_tile_size_and_mode(tmp_path):
    code = "import sys\n" + CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"), tmp=str(tmp_path), runs=RUNS)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, NETFLUX_B200_DEBUG="1"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "debug ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
    space = {}
    exec(RUNS, space)
    for name, U in space["runs"]():
        assert np.array_equal(U, np.load(tmp_path / (name + ".npy"))), name
