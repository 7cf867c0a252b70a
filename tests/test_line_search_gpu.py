"""The inversion driver's line search and misfit with parts of the driver replaced: every
override (a ray object's forward model, a method set on the instance, the policy's clamp) is
used for the trials too, and what the misfit formula takes -- weights that broadcast, a ray
object with the two methods of the reference alone -- is taken."""
import os

import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine.inversion import AdjointStateInversion

pytestmark = pytest.mark.gpu


class _Obj:
    def __init__(self, **kw):
        self.__dict__.update(kw)


@pytest.fixture
def golden(golden_dir):
    z = dict(np.load(os.path.join(golden_dir, "inversion_small.npz")))
    nx, ny, nz = (int(v) for v in z["n"])
    d = float(z["d"])

    def model():
        return _Obj(nx=nx, ny=ny, nz=nz, dx=d, dy=d, dz=d, origin_x=0.0, origin_y=0.0, origin_z=0.0,
                    vp=z["vp0"].copy(), vp_min=1450.0, vp_max=8500.0)

    def rays(cls=se.rays.SampledRays):
        n = z["travel_time"].size
        return cls(model(), z["src_xyz"], z["sta_xyz"], z["weight"], np.ones(n, np.uint8),
                   np.sqrt(((z["src_xyz"] - z["sta_xyz"]) ** 2).sum(axis=1)))

    return _Obj(z=z, model=model, rays=rays)


def _driver(golden, cls=AdjointStateInversion, rays=None, **kw):
    z = golden.z
    args = dict(max_iterations=3, step_length=float(z["step_length"]), smoothing_sigma=float(z["smoothing_sigma"]),
                regularization_lambda=float(z["regularization_lambda"]), misfit_type="l2", line_search_max=3,
                observed=z["travel_time"], weights=z["weight"])
    args.update(kw)
    return cls(golden.model(), _Obj(), None, rays=golden.rays() if rays is None else rays, **args)


def _search(driver):
    """Three trials, none accepted."""
    vp = driver._vp_device()
    g = torch.linspace(-1.0, 1.0, vp.numel(), dtype=torch.float64, device=vp.device)
    return driver._line_search(vp, g, -1.0)


class _Bent(se.rays.SampledRays):
    calls = 0

    def forward_model(self, vp, out=None):
        self.calls += 1
        return super().forward_model(vp, out) * 1.02


class _TwoMethods:
    """The reference's two methods and nothing else."""

    def __init__(self, rays):
        self._rays = rays
        self.calls = 0

    def forward_model(self, vp):
        self.calls += 1
        return self._rays.forward_model(vp)

    def compute_gradient(self, vp, residuals):
        return self._rays.compute_gradient(vp, residuals)


class _Unfused(AdjointStateInversion):
    def _forward(self, vp):
        return self.rays.forward_model(vp)


def test_trials_use_the_rays_own_forward_model(golden):
    a, b = golden.rays(_Bent), golden.rays(_Bent)
    steps = [[], []]
    res = [_driver(golden, rays=a).run(callback=lambda i, m, g, s: steps[0].append(s)),
           _driver(golden, _Unfused, rays=b).run(callback=lambda i, m, g, s: steps[1].append(s))]
    assert a.calls == b.calls > len(steps[0])
    assert steps[0] == steps[1]
    np.testing.assert_array_equal(res[0]["misfit_history"], res[1]["misfit_history"])


@pytest.mark.parametrize("what", ["_forward", "_misfit", "_l1", "rays.forward_model", "rays.misfit",
                                  "fault_policy.clamp_velocity"])
def test_trials_use_what_is_set_on_the_instance(golden, what):
    driver = _driver(golden)
    step = _search(driver)
    owner = driver
    *path, name = what.split(".")
    for p in path:
        owner = getattr(owner, p)
    stock, calls = getattr(owner, name), []

    def counted(*a, **kw):
        calls.append(name)
        return stock(*a, **kw)

    setattr(owner, name, counted)
    assert _search(driver) == step
    assert len(calls) == 3


def test_trials_of_a_foreign_method(golden):
    driver, other = _driver(golden), _driver(golden, rays=golden.rays(_Bent))
    driver._forward = other._forward  # the same function, bound to another driver
    _search(driver)
    assert other.rays.calls == 3


@pytest.mark.parametrize("misfit", ["l2", "l1"])
def test_weights_that_broadcast(golden, misfit):
    n = golden.z["travel_time"].size
    want = _driver(golden, weights=np.full(n, 0.5), misfit_type=misfit).run()
    got = _driver(golden, weights=0.5, misfit_type=misfit).run()
    np.testing.assert_allclose(got["misfit_history"], want["misfit_history"], rtol=1e-12)


def test_rays_with_the_two_methods_alone(golden):
    rays = _TwoMethods(golden.rays())
    want, got = _driver(golden).run(), _driver(golden, rays=rays).run()
    np.testing.assert_allclose(got["misfit_history"], want["misfit_history"], rtol=1e-12)
    assert rays.calls > len(got["misfit_history"])


def test_ranges_out_of_order_end_at_the_upper_bound(golden):
    """clamp(lo, hi) with lo > hi is hi, whichever way the trial is formed."""
    out = []
    for cls in (AdjointStateInversion, _Unfused):
        driver = _driver(golden, cls)
        driver.model.vp_min, driver.model.vp_max = 4000.0, 2000.0
        vp = driver._vp_device()
        at2000 = driver._misfit(driver._forward(torch.full_like(vp, 2000.0)))
        driver.line_search_max = 1
        zero = torch.zeros_like(vp)
        out.append([driver._line_search(vp, zero, at2000 * (1 + 1e-9)), driver._line_search(vp, zero, at2000 * (1 - 1e-9))])
        assert out[-1] == [driver.step_length, driver.step_length * driver.line_search_factor]
    assert out[0] == out[1]


def test_unknown_misfit_is_refused(golden):
    with pytest.raises(ValueError):
        _driver(golden, misfit_type="huber").run()
