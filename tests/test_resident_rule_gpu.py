"""Which small grids keep a forward shot on the SMs: blocks that receive their halo rows in one to
three rounds do, in four or more do not (launches of two steps). Either way seismograms and fields
are bit for bit those of one step per launch. The launch counts tell the paths apart."""
import ctypes

import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu
NT = 13


def _launches():
    n = ctypes.c_longlong()
    call("st_launch_count", ctypes.byref(n))
    return n.value


def _shot(s, n, wav, rec):
    seis = torch.full((NT, rec.count), 7.0, device="cuda")
    before = _launches()
    se.shot_forward(s, (n[0] // 2, n[1] // 3, n[2] - 2), wav, NT, rec, seis=seis)
    torch.cuda.synchronize()
    return _launches() - before, seis.cpu().numpy(), s.get_field(0), s.get_field(1)


@pytest.mark.parametrize("n,resident", [
    ((40, 40, 320), True),    # one round
    ((12, 12, 1200), True),   # two: one row and one plane per block
    ((20, 20, 1000), True),
    ((40, 40, 500), True),    # three
    ((36, 36, 499), True),
    ((33, 18, 700), False),   # four
    ((14, 14, 2040), False),
    ((50, 50, 499), False),   # six
    ((20, 20, 1300), False),  # eight
])
@pytest.mark.parametrize("sponge", ["reference", "stable"])
def test_rule(monkeypatch, n, resident, sponge):
    nx, ny, nz = n
    dt = se.workloads.cfl_dt(10.0, 3000.0)
    s = se.WaveEquationSolver(se.GridParams(nx, ny, nz, 10.0, 10.0, 10.0),
                              se.SolverConfig(dt=dt, nt=NT, sponge_width=3, sponge_damping=0.02))
    s.set_sponge_mode(sponge)
    vel = 1500.0 + 1500.0 * np.random.default_rng(3).random(n)
    s.set_velocity_field(se.workloads.to_reference_layout(vel))
    rec = se.workloads.ReceiverGrid(1, 3, (nx + 1) // 3, 0, 2, (ny + 1) // 2, nz - 3)
    wav = se.workloads.ricker(30.0, dt, NT) + 1e-3
    _shot(s, n, wav, rec)  # the coefficients are formed
    got = _shot(s, n, wav, rec)
    s.set_step_fusion(1)
    one = _shot(s, n, wav, rec)
    s.set_step_fusion(2)
    monkeypatch.setenv("SEISMIC_GB300_XCHUNKS", "3")
    two = _shot(s, n, wav, rec)
    s.close()
    assert (got[0] < two[0]) == resident and two[0] < one[0]
    for a, b, c in zip(one[1:], got[1:], two[1:]):
        assert np.abs(a).max() > 0 and np.array_equal(a, b) and np.array_equal(a, c)
