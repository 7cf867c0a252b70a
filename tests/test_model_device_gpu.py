"""A model set from a device tensor: the host view of it, the time-step rule
and later partial host updates see what a host upload of the same model gives."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine import _lib, fwi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 6, 7), (33, 20, 65)])
@pytest.mark.parametrize("vmax", [3000.0, 14000.0])  # 14000: the CFL damping applies
def test_device_model(shape, vmax):
    rng = np.random.default_rng(shape[2])
    v = rng.uniform(1500.0, vmax, shape).astype(np.float32)
    v.flat[0] = vmax
    if v.size > 3:
        v.flat[1], v.flat[2], v.flat[3] = np.inf, np.nan, -5.0
    pad = np.pad(v.astype(np.float64), 1, mode="edge").reshape(-1)
    dev, host = (se.WaveEquationSolver(se.GridParams(*shape, 10.0, 10.0, 10.0),
                                       se.SolverConfig(dt=0.001, nt=4, sponge_width=0)) for _ in range(2))
    fwi.set_velocity_device(dev, torch.from_numpy(v).cuda())
    host.set_velocity_field(pad)
    assert dev.verify_cfl() == host.verify_cfl()
    np.testing.assert_array_equal(dev.get_field(_lib.ST_FIELD_VELOCITY), pad)
    src = tuple(s // 2 for s in shape)
    for s in (dev, host):
        s.inject_source(*src, [1.0])
        for t in range(4):
            s.step_forward(t)
    np.testing.assert_array_equal(dev.get_field(0), host.get_field(0))
    # a partial host update on top of the device model
    half = np.full(pad.size // 2, 1700.0)
    for s in (dev, host):
        s.set_velocity_field(half)
    np.testing.assert_array_equal(dev.get_field(_lib.ST_FIELD_VELOCITY), host.get_field(_lib.ST_FIELD_VELOCITY))
    assert dev.verify_cfl() == host.verify_cfl()
