"""The trimmed rows of the traversal at their edges, on the device: points on the
faces of cells, neighbours exactly at the search radius and an ulp beyond it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = 0.25


def _points(n):
    """Multiples of 2^-9: on cell faces (the cells are R / 2 or R wide from a bound
    that is a multiple of them) and anywhere, and for each of those one at R along
    an axis. Some of the last are moved on by 2^-23: then |x_ij|^2 is R^2 + 2^-24,
    eight ulps beyond R^2."""
    rng = np.random.Generator(np.random.PCG64(n))
    k = n // 4
    faces = rng.integers(2, 7, (3, k)) / 8.0
    free = rng.integers(128, 385, (3, k)) / 512.0
    base = np.concatenate([faces, free], 1)
    steps = np.array([[128, 0, 0], [0, 128, 0], [0, 0, 128], [-128, 0, 0], [0, -128, 0],
                      [0, 0, -128]]) / 512.0
    at = base + steps[rng.integers(0, 6, 2 * k)].T
    moved = at + np.sign(at - base) * 2.0 ** -23 * (rng.random(2 * k) < 0.3)
    inside = ((moved > 0) & (moved < 1)).all(0)
    return np.concatenate([base, moved[:, inside]], 1).astype(np.float32)


@pytest.mark.parametrize("ratio", [0.5, 1.0])
@pytest.mark.parametrize("order", [0, 1])
def test_neighbours_at_the_radius(cuda, ratio, order):
    import torch

    import reyn_b200 as rb
    p = _points(2000)
    n = p.shape[1]
    grid = rb.Grid((0, 0, 0), (1, 1, 1), R, ratio, order)
    t = [torch.tensor(c, device="cuda") for c in p]
    grid.construct(*t)
    count, len2, _ = grid.neighbour_stats(*t)
    # differences are exact in 32 bits, and no rounding of the squares' sum crosses
    # R^2: pairs at R are exact, those beyond it lie eight ulps away
    d = p.T.astype(np.float64)[:, None] - p.T.astype(np.float64)[None]
    l2 = (d.astype(np.float32).astype(np.float64) ** 2).sum(2).astype(np.float32)
    near = l2 <= np.float32(R * R)
    assert (l2 == np.float32(R * R)).sum() > n // 2
    np.testing.assert_array_equal(count.cpu().numpy(), near.sum(1) - 1)
    want = np.where(near, l2.astype(np.float64), 0.0).sum(1)
    got = len2.cpu().numpy().astype(np.float64)
    assert np.abs(got - want).max() <= 2.0 ** -24 * near.sum(1).max() * want.max()
    grid.close()
