"""The sampled-ray quotients through the cells' reciprocals against the oracle's
divisions, bit for bit, with velocities and distances in and beyond the range
the reciprocal is used for; and the line search's misfits against their
formula in numpy (sums of n terms: n 2^-53)."""
import numpy as np
import pytest
import torch

import seismic_engine as se

pytestmark = pytest.mark.gpu


def _picks(n_cells, n_picks, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    n = np.array([n_cells] * 3)
    d, o = np.full(3, 200.0 * scale), np.zeros(3)
    ext = n_cells * 200.0 * scale
    src, sta = rng.uniform(0, ext, (n_picks, 3)), rng.uniform(0, ext, (n_picks, 3))
    return n, d, o, src, sta, rng.uniform(0.5, 1.5, n_picks), rng


@pytest.mark.parametrize("scale", [1.0, 1e-80, 1e120])
@pytest.mark.parametrize("kind", ["ordinary", "extreme"])
def test_quotients(oracle, kind, scale):
    n, d, o, src, sta, w, rng = _picks(21, 3001, 5, scale)
    vp = rng.uniform(1450.0, 8500.0, 21 ** 3)
    if kind == "extreme":
        some = rng.integers(0, 12, vp.size)
        for k, v in enumerate((1e-310, 1e-200, 1e-95, 1e95, 1e200, 1.7e308, np.inf, np.nan, 0.0, -3.0)):
            vp[some == k] = v
    res = rng.standard_normal(w.size)
    rays = se.SampledRays((*n, *d, *o), src, sta, w)
    vp3 = vp.reshape(21, 21, 21)
    np.testing.assert_array_equal(rays.forward_model(vp), oracle.sampled_traveltimes(n, d, o, src, sta, None, vp3))
    np.testing.assert_array_equal(rays.compute_gradient(vp, res),
                                  oracle.sampled_gradient(n, d, o, src, sta, None, w, vp3, res).reshape(-1))


@pytest.mark.parametrize("l1", [False, True])
@pytest.mark.parametrize("n_picks", [1, 255, 200_001])
def test_trial_misfit(n_picks, l1):
    n, d, o, src, sta, w, rng = _picks(13, n_picks, 7)
    rays = se.SampledRays((*n, *d, *o), src, sta, w)
    vp, g = rng.uniform(1450.0, 8500.0, 13 ** 3), rng.standard_normal(13 ** 3)
    vp[3], g[5] = np.nan, np.inf
    obs = np.abs(rng.standard_normal(n_picks))
    to = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    vd, gd, od, wd = to(vp), to(g), to(obs), to(w)
    for policy in (None, (1500.0, 8000.0)):
        trial = vp - 700.0 * g
        for lo, hi in ([policy] if policy else []) + [(1450.0, 8500.0)]:
            trial = np.clip(np.where(np.isfinite(trial), trial, lo), lo, hi)
        t = rays.forward_model(to(trial))
        r = obs - t.cpu().numpy()
        want = (w * np.abs(r)).sum() if l1 else 0.5 * (w * r * r).sum()
        got = rays.trial_misfit(vd, gd, 700.0, policy, 1450.0, 8500.0, od, wd, l1)
        # the same times give the same bits whichever way they were formed
        assert got == rays.misfit(t, od, wd, l1)
        assert abs(got - want) <= (n_picks + 4) * 2.0 ** -53 * want
    with pytest.raises(ValueError):
        rays.misfit(od[:-1], od, wd)
