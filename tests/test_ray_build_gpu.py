"""The walk-once ray-matrix build against the oracle's traversal and sorted
triplets, bit for bit (row pointers, columns, lengths rounded once to FP32):
every octant, axis-aligned and degenerate rays, rays through grid corners
(ties), starts outside the grid, ranges the fast walk hands over, grids with
long rows and counts around the 32-ray tiles."""
import numpy as np
import pytest

import seismic_engine as se

pytestmark = pytest.mark.gpu


def _rays(kind, shape, n, rng):
    s = np.array(shape, float)
    p, q = rng.uniform(0, s, (n, 3)), rng.uniform(0, s, (n, 3))
    if kind == "corners":  # integer and half-integer end points: ties between the axes
        p, q = np.floor(2 * p) / 2, np.floor(2 * q) / 2
    elif kind == "axes":
        keep = rng.integers(0, 3, n)
        for a in range(3):
            q[:, a] = np.where(keep == a, q[:, a], p[:, a])
        q[::7] = p[::7]  # a point
    elif kind == "outside":
        p, q = rng.uniform(-s, 2 * s, (n, 3)), rng.uniform(-s, 2 * s, (n, 3))
    elif kind == "extreme":
        p[::5, 0], q[::5, 0] = 0.25, 0.25 + 1e-17 * rng.standard_normal(p[::5].shape[0])
        p[1::5, 1], q[1::5, 1] = 1e-310, 3e-310
        q[2::5, 2] = 1e305
        p[3::5, 0] = 1e-200
    return np.concatenate([p, q], axis=1)


@pytest.mark.parametrize("shape", [(7, 33, 70), (40, 1, 3), (1, 1, 1), (300, 5, 260)])
@pytest.mark.parametrize("kind", ["any", "corners", "axes", "outside", "extreme"])
def test_ray_matrix_is_the_oracles(oracle, kind, shape):
    rng = np.random.default_rng(sum(shape) + len(kind))
    for n in (1, 31, 33, 1000):
        ends = _rays(kind, shape, n, rng)
        rp, col, val = oracle.ray_matrix(ends, *shape, h=12.5)
        m = se.CSRMatrix()
        assert m.build_ray_matrix(ends, *shape, cell_size=12.5) == col.size
        np.testing.assert_array_equal(m.row_ptr(), rp)
        np.testing.assert_array_equal(m.col_ind(), col)
        np.testing.assert_array_equal(m.values(), val.astype(np.float32).astype(np.float64))
