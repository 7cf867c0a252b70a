"""The transpose of a matrix whose device columns were rewritten by the caller
(the arrays are handed out writable): entries outside the columns are dropped and
repeated ones are summed, as in a build from triplets."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu


class _Array:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


def _rewritten(cols, change, nnz=6000, seed=3):
    rng = np.random.default_rng(seed)
    rows = 900
    key = np.unique(rng.integers(0, rows * cols, nnz))
    r, c = key // cols, key % cols
    v = rng.integers(1, 5, key.size).astype(np.float64)
    A = se.CSRMatrix().build_from_triplets(rows, cols, r, c, v)
    c = c.copy()
    change(c, r, rng)
    torch.as_tensor(_Array(A.device_arrays()[1], c.size, "<i4"), device="cuda").copy_(torch.from_numpy(c.astype(np.int32)))
    torch.cuda.synchronize()
    return A, rows, r, c, v


def _outside(c, r, rng):
    i = rng.choice(c.size, 200, replace=False)
    c[i] = rng.choice([-1, -7, c.max() + 1, 1 << 20, (1 << 31) - 1, -(1 << 31)], 200)


def _repeated(c, r, rng):
    i = np.flatnonzero(np.diff(r) == 0)[::3]
    c[i + 1] = c[i]


def _shuffled(c, r, rng):
    for a in np.unique(r):  # a row's columns in another order
        i = np.flatnonzero(r == a)
        c[i] = rng.permutation(c[i])


@pytest.mark.parametrize("change", [_outside, _repeated, _shuffled])
@pytest.mark.parametrize("cols", [70, 1100, 3_000_000])
def test_transpose_of_rewritten_columns(cols, change):
    A, rows, r, c, v = _rewritten(cols, change)
    ok = (c >= 0) & (c < cols)
    x = np.random.default_rng(1).integers(-8, 9, rows)
    want = np.zeros(cols)
    np.add.at(want, c[ok], v[ok] * x[r[ok]])
    y, xd = torch.full((cols,), 7.0, device="cuda"), torch.from_numpy(x.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    A.spmv_device(xd, y, transpose=True)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), want)
    # the diagonal of A^T A: repeated entries are one entry of their sum
    cell, inv = np.unique(r[ok] * cols + c[ok], return_inverse=True)
    value = np.bincount(inv, v[ok])
    lam = 1.0
    diag = np.bincount(cell % cols, value ** 2, minlength=cols) + lam
    d = torch.zeros(cols, device="cuda")
    torch.cuda.synchronize()
    call("st_csr_normal_jacobi", A.handle, lam, d.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy(), (1.0 / diag).astype(np.float32))


def test_transpose_with_no_valid_column():
    def none(c, r, rng):
        c[:] = -1
    A, rows, *_ = _rewritten(300, none)
    y = torch.full((300,), 7.0, device="cuda")
    x = torch.ones(rows, device="cuda")
    torch.cuda.synchronize()
    A.spmv_device(x, y, transpose=True)
    torch.cuda.synchronize()
    assert not y.any()
