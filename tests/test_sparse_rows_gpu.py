"""Short-row SpMV, the normal-equation diagonal and the CG vector kernels at
their edges: tiles of 128 rows, tiles with more entries than fit in shared
memory, empty rows, a start that is not 16-byte aligned, an unaligned solution
vector. Reference: FP64 numpy; bounds from FP32 rounding (a row of m entries:
(m + 1) 2^-24 sum |a x|; the squares' sums and their inverse: 2^-23)."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine import _lib
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _matrix(lengths, cols, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lengths)])
    col = np.concatenate([np.sort(rng.choice(cols, m, replace=False)) for m in lengths] + [np.zeros(0, np.int64)])
    val = rng.standard_normal(rp[-1]).astype(np.float32)
    rows = np.repeat(np.arange(len(lengths)), lengths)
    A = se.CSRMatrix().build_from_triplets(len(lengths), cols, rows, col, val.astype(np.float64))
    return A, rp, col.astype(np.int64), val


def _lengths(kind, rows, rng):
    if kind == "seven":
        return np.full(rows, 7)
    if kind == "mixed":
        return rng.integers(0, 12, rows)
    m = rng.integers(0, 5, rows)
    m[rows // 2] = 3000  # one row beyond the shared-memory tile
    return m


@pytest.mark.parametrize("kind", ["seven", "mixed", "long"])
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 255, 256, 257, 5003])
def test_short_rows(kind, rows):
    rng = np.random.default_rng(rows)
    lengths = _lengths(kind, rows, rng)
    if kind == "long" and rows < 1000:
        lengths = np.minimum(lengths, 9)
    A, rp, col, val = _matrix(lengths, 4000, rows)
    x = rng.standard_normal(4000).astype(np.float32)
    xd, y = torch.from_numpy(x).cuda(), torch.zeros(rows, device="cuda")
    torch.cuda.synchronize()
    A.spmv_device(xd, y)
    torch.cuda.synchronize()
    prod = val.astype(np.float64) * x[col]
    want = np.array([prod[a:b].sum() for a, b in zip(rp[:-1], rp[1:])])
    mag = np.array([np.abs(prod[a:b]).sum() for a, b in zip(rp[:-1], rp[1:])])
    assert np.all(np.abs(y.cpu().numpy() - want) <= (lengths + 1) * EPS * mag)


@pytest.mark.parametrize("scale", [1.0, 1e-22, 1e22])  # 1e-22, 1e22: the squares leave the FP32 range
@pytest.mark.parametrize("rows,m", [(3, 1), (700, 6), (130, 40), (1000, 300), (40_000, 300)])
def test_normal_diagonal(rows, m, scale):
    A, rp, col, val = _matrix(np.full(rows, m), 500, m)
    A.scale(scale)
    val = val * np.float32(scale)
    d = torch.zeros(500, device="cuda")
    torch.cuda.synchronize()
    lam = 0.25 * scale * scale
    call("st_csr_normal_jacobi", A.handle, lam, d.data_ptr())
    torch.cuda.synchronize()
    want = 1.0 / (np.bincount(col, val.astype(np.float64) ** 2, minlength=500) + lam)
    got = d.cpu().numpy()
    fits = want < 3.4e38
    # the reference as the output's type holds it (at 1e22 the inverses are subnormal)
    np.testing.assert_allclose(got[fits], want[fits].astype(np.float32), rtol=2 * EPS)
    assert np.isinf(got[~fits]).all()


@pytest.mark.parametrize("scale", [1.0, 1e-15, 1e25, 1e-25])
def test_cg_scales_with_its_right_hand_side(scale):
    """Residuals at and beyond the range of the FP32 pairs: the iterates follow the right-hand side's scale, down to
    the solver's own stop at |p.q| < 1e-30."""
    n = 4100
    idx = np.arange(n)
    diag = 2.0 + np.random.default_rng(n).random(n)
    A = se.CSRMatrix().build_from_triplets(n, n, np.concatenate([idx, idx[1:]]), np.concatenate([idx, idx[:-1]]),
                                           np.concatenate([diag, np.full(n - 1, -0.5)]))
    b = torch.from_numpy(np.random.default_rng(n + 1).standard_normal(n).astype(np.float32)).cuda()
    x, xs = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    se.normal_cg_device(A, None, 0.1, x, 3, 1e-30, True, rhs=b)
    it, rel, _ = se.normal_cg_device(A, None, 0.1, xs, 3, 1e-30, True, rhs=b * scale)
    if scale == 1e-25:
        assert it == 0 and not xs.any()
        return
    assert it == 3 and 0.0 < rel < 1.0
    # b * scale rounds once per value, then the iterations' own rounding
    np.testing.assert_allclose(xs.double().cpu().numpy() / scale, x.double().cpu().numpy(), rtol=0,
                               atol=64 * EPS * float(x.abs().max()))


@pytest.mark.parametrize("n", [1, 5, 1026, 70001])
def test_cg_on_an_unaligned_solution(n):
    """The same iterates with x on a 16-byte boundary (quads) and off it (single words)."""
    diag = 2.0 + np.random.default_rng(n).random(n)
    idx = np.arange(n)
    A = se.CSRMatrix().build_from_triplets(n, n, np.concatenate([idx, idx[1:]]), np.concatenate([idx, idx[:-1]]),
                                           np.concatenate([diag, np.full(n - 1, -0.5)]))
    b = torch.from_numpy(np.random.default_rng(n + 1).standard_normal(n).astype(np.float32)).cuda()
    out = []
    for off in (0, 1):
        x = torch.zeros(n + 8, device="cuda")[off:off + n]
        se.normal_cg_device(A, None, 0.1, x, 6, 1e-30, True, rhs=b)
        out.append(x.cpu().numpy())
    # the inner products are summed in FP64 in another order: the step lengths agree to a last bit or so
    np.testing.assert_allclose(out[0], out[1], rtol=0, atol=64 * EPS * np.abs(out[0]).max())
    assert np.isfinite(out[0]).all() and _lib.ST_CG_JACOBI
