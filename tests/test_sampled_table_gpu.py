"""The sampled forward model through the table of reciprocals (many samples) and by division (few, or
many cells): the same picks in one object and in sixteen, both against the oracle, bit for bit, with
velocities and distances in and beyond the range the reciprocal is used for."""
import numpy as np
import pytest

import seismic_engine as se

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-80, 1e120])
@pytest.mark.parametrize("kind", ["ordinary", "extreme"])
def test_table_and_division(oracle, kind, scale):
    cells, picks = 21, 250_000
    rng = np.random.default_rng(9)
    n, d, o = np.array([cells] * 3), np.full(3, 200.0 * scale), np.zeros(3)
    src, sta = rng.uniform(0, cells * 200.0 * scale, (2, picks, 3))
    w = np.ones(picks)
    vp = rng.uniform(1450.0, 8500.0, cells ** 3)
    if kind == "extreme":
        some = rng.integers(0, 12, vp.size)
        for k, v in enumerate((1e-310, 1e-200, 1e-95, 1e95, 1e200, 1.7e308, np.inf, np.nan, 0.0, -3.0)):
            vp[some == k] = v
    rays = se.SampledRays((*n, *d, *o), src, sta, w)
    assert rays.n_samples > 400_000 + 9 * cells ** 3 // 4  # the table's side of the line
    want = oracle.sampled_traveltimes(n, d, o, src, sta, None, vp.reshape(cells, cells, cells))
    np.testing.assert_array_equal(rays.forward_model(vp), want)
    for part in np.array_split(np.arange(picks), 16):
        few = se.SampledRays((*n, *d, *o), src[part], sta[part], w[part])
        np.testing.assert_array_equal(few.forward_model(vp), want[part])
