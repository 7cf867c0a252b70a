"""The counting-sort transpose against numpy, at the edges of its tiles (4096
entries), of its digits (1024 bins; one, two and three passes) and of its
ranges. Small integers: every FP32 sum is exact, so products agree bit for bit."""
import numpy as np
import pytest
import torch

import seismic_engine as se

pytestmark = pytest.mark.gpu


def _check(A, rows, cols, r, c, v, seed):
    x = np.random.default_rng(seed).integers(-8, 9, rows)
    want = np.zeros(cols)
    np.add.at(want, c, v * x[r])
    y = torch.full((max(cols, 1),), 7.0, device="cuda")
    xd = torch.from_numpy(x.astype(np.float32)).cuda()
    torch.cuda.synchronize()
    A.spmv_device(xd, y, transpose=True)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy()[:cols], want)


@pytest.mark.parametrize("cols", [1, 2, 1024, 1025, (1 << 20) + 3])
@pytest.mark.parametrize("nnz", [1, 4095, 4097, 300_001])
def test_transpose(cols, nnz):
    rng = np.random.default_rng(cols + nnz)
    rows = 997 if cols > 1000 else max(1, nnz // max(1, cols // 2 + 1)) * 3
    key = np.unique(rng.integers(0, rows * cols, nnz))
    r, c = key // cols, key % cols
    v = rng.integers(1, 5, key.size).astype(np.float64)
    A = se.CSRMatrix().build_from_triplets(rows, cols, r, c, v)
    assert A.nnz() == key.size
    _check(A, rows, cols, r, c, v, nnz)


def test_transpose_of_a_padded_matrix_and_of_none():
    rng = np.random.default_rng(2)
    key = np.unique(rng.integers(0, 50 * 60, 700))
    r, c, v = key // 60, key % 60, rng.integers(1, 5, key.size).astype(np.float64)
    _check(se.CSRMatrix().build_from_triplets(50, 60, r, c, v, pad=True), 50, 60, r, c, v, 3)
    e = np.zeros(0, np.int64)
    _check(se.CSRMatrix().build_from_triplets(5, 9, e, e, e.astype(float)), 5, 9, e, e, e, 4)
    _check(se.CSRMatrix(5, 9, 12), 5, 9, e, e, e, 5)  # declared entries, none in any row


def test_empty_rows_and_one_full_column():
    rows = 20_000
    r = np.arange(0, rows, 3)
    _check(se.CSRMatrix().build_from_triplets(rows, 3000, r, np.full(r.size, 2999), np.ones(r.size)), rows, 3000, r,
           np.full(r.size, 2999), np.ones(r.size), 6)
