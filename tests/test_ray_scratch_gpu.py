"""Ray matrices whose walk-once scratch cannot be allocated: rays whose end
points allow thousands of cells but which leave the grid in their first one ask
for more scratch than the device has, and are built from triplets instead."""
import numpy as np
import pytest
import torch

import seismic_engine as se

pytestmark = pytest.mark.gpu


def test_scratch_beyond_the_device_memory():
    nx, ny, nz, h = 2, 2, 24_000, 12.5
    per_tile = nz * 256  # bytes: at least nz rows of 32 entries of 8 bytes
    total = torch.cuda.get_device_properties(0).total_memory
    n = 32 * (int(1.1 * total) // per_tile + 1)
    if n > 4_000_000:
        pytest.skip("sizes are chosen for devices of up to 700 GB")
    ends = np.tile([0.25, 0.5, 0.5, -1e6, 0.5, nz - 0.5], (n, 1))
    ends[1::2, 1] = ends[1::2, 4] = 1.5
    A = se.CSRMatrix()
    assert A.build_ray_matrix(ends, nx, ny, nz, h) == n
    # one entry each: a quarter of a cell along x, the ray's length at that share
    t = 0.25 / (1e6 + 0.25)
    length = np.sqrt((1e6 + 0.25) ** 2 + (nz - 1.0) ** 2) * t * h
    assert np.array_equal(A.row_ptr(), np.arange(n + 1))
    assert np.array_equal(A.col_ind(), np.where(np.arange(n) % 2 == 0, 0, nz))
    np.testing.assert_allclose(A.values(), length, rtol=2.0 ** -23)
