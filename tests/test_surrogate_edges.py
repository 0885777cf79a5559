"""Ragged and extreme sizes of the surrogate's kernels: batches around the 128-row tiles and the
32-row weight-gradient chunks (and more chunks than the three buffers), and the wall distance's
clusters of 32 points and groups of 1024."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 128, 257, 4737, 148 * 32 * 3 + 5])
def test_gradients_at_ragged_batches(n):
    """Every gradient block within the BF16 bound of the other gradient test (3e-2 relative L2: each
    activation and weight carries 2^-9, a few of them in sequence)."""
    from netflux_b200 import surrogate as sur
    m = sur.MLP(seed=5)
    rng = np.random.default_rng(n)
    f = rng.uniform(-1, 1, (n, 7)).astype(np.float32)
    t = rng.normal(0, 0.5, (n, 5)).astype(np.float32)
    loss, g = m.gradients(f, t)
    lo, go = mo.loss_and_grad(m.get_params(), f, t)
    assert abs(loss - lo) <= 1e-3 * lo
    for a, b in ((mo.OFF_W0, mo.OFF_W1), (mo.OFF_W1, mo.OFF_W2), (mo.OFF_W2, mo.OFF_W3), (mo.OFF_W3, mo.OFF_B1),
                 (mo.OFF_B1, mo.OFF_W4), (mo.OFF_W4, mo.OFF_B4), (mo.OFF_B4, mo.N_PARAM)):
        assert np.linalg.norm(g[a:b] - go[a:b]) <= 3e-2 * max(np.linalg.norm(go[a:b]), 1e-30)
    y, _ = m.predict(f)
    yo, _ = mo.forward(m.get_params(), f)
    assert np.abs(y - yo).max() <= 2e-2 * np.abs(yo).max()


def _wall(points, wall):
    from netflux_b200 import _lib as L
    out = np.empty(points.shape[0], np.float32)
    assert L.load().nf_wall_distance(L.fptr(points), points.shape[0], L.fptr(wall), wall.shape[0], L.fptr(out)) == L.NF_OK
    return out


@pytest.mark.parametrize("n", [1, 31, 257, 3001])
@pytest.mark.parametrize("m", [1, 31, 32, 33, 1023, 1025, 5000, 40000])
def test_wall_distance_is_the_minimum_over_all_points(n, m):
    """Against FP64 brute force (each FP32 distance within 4 roundings of 2^-24), and the same bits for
    points and wall points in any order, which pass over different boxes."""
    rng = np.random.default_rng(n * 100000 + m)
    # points on the faces of a box in rows, and points inside and around it
    wall = rng.uniform(0, 1, (m, 3)).astype(np.float32)
    wall[np.arange(m), rng.integers(0, 3, m)] = rng.integers(0, 2, m)
    wall = wall[np.lexsort((wall[:, 0], wall[:, 1], wall[:, 2]))].copy()
    pts = rng.uniform(-0.2, 1.2, (n, 3)).astype(np.float32)
    pts[: min(n, 5)] = wall[: min(n, 5)] if m >= 5 or n <= m else pts[: min(n, 5)]
    d = _wall(pts, wall)
    ref = np.array([np.sqrt(((wall.astype(np.float64) - p.astype(np.float64)) ** 2).sum(1).min()) for p in pts])
    assert np.abs(d - ref).max() <= 4 * 2.0 ** -24 * max(ref.max(), 1.0)
    pw, pp = rng.permutation(m), rng.permutation(n)
    assert np.array_equal(_wall(pts, wall[pw].copy()), d)
    assert np.array_equal(_wall(pts[pp].copy(), wall), d[pp])
