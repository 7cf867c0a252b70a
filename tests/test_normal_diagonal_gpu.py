"""The normal-equation diagonal by groups of 8, 16 and 32 lanes per row: mean lengths on either side of
each choice, row counts that leave groups and warps without rows, rows beyond what a lane's triple holds
(256 products), one row that needs FP64 beside others that do not, and sums on either side of 2^-40,
below which FP64 takes over. Reference: FP64 numpy; the sums
are no less precise, so the inverse is off by its rounding to FP32 alone (2^-23)."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [24, 159, 160, 479, 480])
@pytest.mark.parametrize("columns", [1, 3, 33, 1000])
@pytest.mark.parametrize("kind", ["even", "uneven", "large", "tiny"])
def test_diagonal(mean, columns, kind):
    rng = np.random.default_rng(mean + columns)
    m = np.full(columns, mean)
    if kind == "uneven":
        m = np.arange(columns) % (2 * mean + 1)
        m[0] += mean * columns - m.sum() + columns  # thousands of entries in one column
    val = rng.standard_normal(m.sum()).astype(np.float32)
    if kind == "large":
        val[-1] = 2.0 ** 62
    lam = 0.25
    if kind == "tiny":
        val *= np.float32(2.0 ** -20 / np.sqrt(mean))
        val[::3] *= np.float32(2.0 ** -60)
        lam = 0.0
    col = np.repeat(np.arange(columns), m)
    row = np.concatenate([np.arange(n) for n in m])
    A = se.CSRMatrix().build_from_triplets(int(m.max()), columns, row, col, val.astype(np.float64))
    d = torch.zeros(columns, device="cuda")
    torch.cuda.synchronize()
    call("st_csr_normal_jacobi", A.handle, lam, d.data_ptr())
    torch.cuda.synchronize()
    want = 1.0 / (np.bincount(col, val.astype(np.float64) ** 2, minlength=columns) + lam)
    np.testing.assert_allclose(d.cpu().numpy(), want, rtol=2.0 ** -23)
