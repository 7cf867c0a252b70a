"""Sums of products at the edges of the FP32 triples that carry them: the
normal-equation diagonal (both kernels) where the squares' sum leaves the FP32
range and where it needs all of FP64's bits, the CG residual likewise, and the
short-row product where one rounding a term shows. Every expected value is exact."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu


def _matrix(columns, rows, fill):
    """columns: the entries of the first columns; 100 more columns of `fill` ones (their mean picks the kernel)."""
    r, c, v = [], [], []
    for j, entries in enumerate(columns + [np.ones(fill)] * 100):
        r.append(np.arange(len(entries)))
        c.append(np.full(len(entries), j))
        v.append(np.asarray(entries, np.float64))
    cols = len(columns) + 100
    return se.CSRMatrix().build_from_triplets(rows, cols, np.concatenate(r), np.concatenate(c), np.concatenate(v)), cols


def _diagonal(A, cols, lam):
    d = torch.zeros(cols, device="cuda")
    torch.cuda.synchronize()
    call("st_csr_normal_jacobi", A.handle, lam, d.data_ptr())
    torch.cuda.synchronize()
    return d.cpu().numpy()


@pytest.mark.parametrize("fill", [2, 60])
@pytest.mark.parametrize("power", [46, 50, 51, 58, 60, 61])
def test_diagonal_of_large_entries(power, fill):
    """Sums of 2^8 .. 2^14 squares up to 2^128 and beyond: the inverse, subnormal at the top, is a power of two."""
    counts = (255, 256, 257, 300, 4096, 9000)
    A, cols = _matrix([np.full(m, 2.0 ** power) for m in counts], 9000, fill)
    want = np.float32(1.0 / (np.array(counts, np.float64) * 4.0 ** power))
    assert np.array_equal(_diagonal(A, cols, 0.0)[:len(counts)], want)


@pytest.mark.parametrize("fill", [2, 60])
def test_diagonal_keeps_every_bit_of_fp64(fill):
    # squares 2^24 + 1 + 4 * 2^-28, 53 bits in any order of summation; lam leaves the last
    A, cols = _matrix([[2.0 ** 12, 1.0] + [2.0 ** -14] * 4], 100, fill)
    assert _diagonal(A, cols, -(2.0 ** 24 + 1.0))[0] == 2.0 ** 26


def test_cg_residual_keeps_every_bit_of_fp64():
    # r = b / 2 after one step with alpha = 1/2 (diagonal 1 and 3 in equal parts); the squares of a quad
    # need 52 bits, and so do the sums of 32 equal quads
    n = 128
    diag = np.where(np.arange(n) < n // 2, 1.0, 3.0)
    A = se.CSRMatrix().build_from_triplets(n, n, np.arange(n), np.arange(n), diag)
    b = np.tile([2.0 ** 13, 2.0, 1.5 * 2.0 ** -12, 1.5 * 2.0 ** -12], n // 4)
    se.SparseOps.conjugate_gradient(A, b, 1, 1e-30)
    assert se.SparseOps.last_iterations == 1
    assert se.SparseOps.last_relative_residual == 0.5


@pytest.mark.parametrize("lengths", [[9] * 300, [9] * 7 + [3] * 290])
def test_short_row_products_are_fused(lengths):
    # the ninth entry cancels the first to 2^-46, which a product rounded before the addition loses
    rows, cols = len(lengths), 200
    r = np.repeat(np.arange(rows), lengths)
    k = np.concatenate([np.arange(m) for m in lengths])
    e = 2.0 ** -23
    v = np.where(k == 0, 1.0, np.where(k == 8, -(1.0 - e), 0.0))
    x = np.zeros(cols, np.float32)
    x[0], x[8] = 1.0, 1.0 + e
    A = se.CSRMatrix().build_from_triplets(rows, cols, r, k, v)
    xd, y = torch.from_numpy(x).cuda(), torch.zeros(rows, device="cuda")
    torch.cuda.synchronize()
    A.spmv_device(xd, y)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), np.where(np.array(lengths) > 8, np.float32(e * e), np.float32(1.0)))
