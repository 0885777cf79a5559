"""The wall distance with points and wall points in order, where boxes are passed over, and in none,
where a block compares all pairs: the same bits, over part tiles of 1024 wall points and part blocks."""
import numpy as np
import pytest

from test_surrogate_edges import _wall

pytestmark = pytest.mark.gpu


def _lattice(n, hi):
    a = [np.linspace(0, e, k) for k, e in zip(n, hi)]
    return np.stack(np.meshgrid(*a, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)


@pytest.mark.parametrize("n", [(1, 1, 1), (3, 5, 17), (16, 16, 16), (33, 21, 30)])
@pytest.mark.parametrize("m", [(1, 40), (30, 35), (64, 80), (100, 101)])
def test_order_changes_no_bit(n, m):
    points, wall = _lattice(n, (1, 1, 1)), _lattice((m[0], 1, m[1]), (1, 0, 1))
    rng = np.random.default_rng(sum(n) + sum(m))
    d = _wall(points, wall)
    pp, pw = rng.permutation(len(points)), rng.permutation(len(wall))
    half = np.arange(len(points))
    half[: len(points) // 2] = rng.permutation(len(points) // 2)
    assert np.array_equal(_wall(points[pp].copy(), wall), d[pp])
    assert np.array_equal(_wall(points, wall[pw].copy()), d)
    assert np.array_equal(_wall(points[pp].copy(), wall[pw].copy()), d[pp])
    assert np.array_equal(_wall(points[half].copy(), wall), d[half])
    few = rng.choice(len(points), min(200, len(points)), replace=False)
    ref = np.array([np.sqrt(((wall.astype(np.float64) - points[i].astype(np.float64)) ** 2).sum(1).min()) for i in few])
    assert np.abs(d[few] - ref).max() <= 4 * 2.0 ** -24  # four roundings of a distance of at most 1


@pytest.mark.parametrize("ordered", [True, False])
def test_not_a_number_and_infinity(ordered):
    """A wall point that is not a number is passed over; a point that is not a number, or infinitely far,
    gets the largest distance; the others' are as without them."""
    points, wall = _lattice((8, 8, 9), (1, 1, 1)), _lattice((50, 1, 50), (1, 0, 1))
    if not ordered:
        rng = np.random.default_rng(2)
        points, wall = points[rng.permutation(len(points))].copy(), wall[rng.permutation(len(wall))].copy()
    keep = np.ones(len(wall), bool)
    keep[[0, 777, len(wall) - 1]] = False
    d = _wall(points, wall[keep].copy())
    wall[~keep, 1] = np.nan
    points[[3, 300], 0] = np.nan, np.inf
    out = _wall(points, wall)
    others = np.ones(len(points), bool)
    others[[3, 300]] = False
    assert np.array_equal(out[others], d[others])
    assert (out[~others] == np.sqrt(np.float32(3.0e38))).all()
