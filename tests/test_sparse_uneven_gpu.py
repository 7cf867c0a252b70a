"""Short-row products whose rows are uneven (groups of lanes per row in place of the
row tiles): 128-row tiles beyond shared memory, tiles with one long row, single rows of
thousands, and the transposes and copies of such matrices. Reference: FP64 numpy; a row
of m entries is off by at most (m + 1) 2^-24 sum |a x| (FP32 fused multiply-adds)."""
import numpy as np
import pytest
import torch

import seismic_engine as se

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24
ROWS = 1500


def _lengths(kind):
    i = np.arange(ROWS)
    return {
        "half": np.where(i < ROWS // 2, 0, 18),                  # four lanes
        "half thin": np.where(i < ROWS // 4, 13, 1),             # two lanes
        "one of 128": np.where(i % 128 == 7, 600, 3),            # four lanes
        "last row": np.where(i == ROWS - 1, 1024, 3),            # two lanes, the longest they take
        "a long row": np.where(i == 3, 1025, 3),                 # row tiles
        "few": np.where(i == 5, 1000, 2),                        # row tiles: fewer than 4,096 entries
        "long rows": np.where(i < 8, 1100, 3),                   # eight lanes: one tile of 9,160 entries
        "sorted": np.sort(np.random.default_rng(2).zipf(1.7, ROWS).clip(0, 3000))[::-1],
    }[kind].astype(np.int64)


def _product(A, x, rows, transpose=False):
    y = torch.zeros(rows, device="cuda")
    torch.cuda.synchronize()
    A.spmv_device(x, y, transpose=transpose)
    torch.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("kind", ["half", "half thin", "one of 128", "last row", "a long row", "few", "long rows", "sorted"])
def test_uneven_rows(kind):
    rng = np.random.default_rng(1)
    m = _lengths(kind)
    cols = 4000
    rp = np.concatenate([[0], np.cumsum(m)])
    col = np.concatenate([np.sort(rng.choice(cols, n, replace=False)) for n in m])
    row = np.repeat(np.arange(ROWS), m)
    val = rng.standard_normal(rp[-1]).astype(np.float32)
    A = se.CSRMatrix().build_from_triplets(ROWS, cols, row, col, val.astype(np.float64))
    T = se.CSRMatrix().build_from_triplets(cols, ROWS, col, row, val.astype(np.float64))
    x = rng.standard_normal(cols).astype(np.float32)
    prod = val.astype(np.float64) * x[col]
    want = np.bincount(row, prod, minlength=ROWS)
    bound = (m + 1) * EPS * np.bincount(row, np.abs(prod), minlength=ROWS)
    xd = torch.from_numpy(x).cuda()
    got = _product(A, xd, ROWS)
    assert np.all(np.abs(got - want) <= bound)
    assert np.array_equal(_product(A.clone(), xd, ROWS), got)
    assert np.all(np.abs(_product(T, xd, ROWS, transpose=True) - want) <= bound)
