"""The tile lists of the stage kernel (build_tiles, netflux_b200/csrc/tiles.cpp), on the host: every code
leads back to the neighbour, boundary face or vertex it stands for, over sizes around the tiles' and
orders from well-kept to random, also where the system grants fewer threads than asked for."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = [os.path.join(ROOT, "tests", "tiles_check.cpp")] + [
    os.path.join(ROOT, "netflux_b200", "csrc", f) for f in ("tiles.cpp", "mesh.cpp")]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("tiles") / "tiles_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, *SRC, "-ldl", "-pthread"], check=True)

    def run(*args, **env):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, **env))
        assert r.returncode == 0 and "tiles ok" in r.stdout, (args, r.returncode, r.stdout[-500:], r.stderr[-500:])
    return run


@pytest.mark.parametrize("tile", [64, 128, 256])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 255, 256, 257, 1000, 20011])
def test_lists_lead_back_to_the_mesh(check, tile, n):
    for spread in (20, 300, 10 ** 6):
        check(n, tile, spread, n + tile, -1)


@pytest.mark.parametrize("granted", [-1, 0, 2])
def test_fewer_threads_than_asked_for(check, granted):
    check(70001, 256, 200, 5, granted, NETFLUX_B200_HOST_THREADS="8")
