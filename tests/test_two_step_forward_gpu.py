"""Forward shots without snapshots by launches of two steps, on grids that a resident shot would take
otherwise (a fixed chunking selects the launches) and on grids that do not fit: both sponge rules, rows
of a multiple of four values and ragged ones, odd and even step counts. Bit for bit one step per launch:
seismograms and the last two fields. The launch counts show that the pairs ran."""
import ctypes

import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu


def _launches():
    n = ctypes.c_longlong()
    call("st_launch_count", ctypes.byref(n))
    return n.value


@pytest.mark.parametrize("sponge", ["reference", "stable"])
@pytest.mark.parametrize("n,nt,chunks", [
    ((30, 20, 36), 12, "3"), ((30, 20, 36), 13, "1"), ((24, 31, 44), 8, "5"), ((17, 33, 64), 11, "17"),
    ((30, 20, 37), 12, "3"), ((24, 31, 45), 11, "2"), ((9, 40, 130), 8, "1"), ((21, 18, 63), 9, "4"),
    ((160, 160, 160), 8, None), ((160, 150, 163), 9, None), ((33, 18, 700), 8, None)])
def test_pairs(monkeypatch, n, nt, chunks, sponge):
    nx, ny, nz = n
    dt = se.workloads.cfl_dt(10.0, 3000.0)
    s = se.WaveEquationSolver(se.GridParams(nx, ny, nz, 10.0, 10.0, 10.0),
                              se.SolverConfig(dt=dt, nt=nt, sponge_width=4, sponge_damping=0.02))
    s.set_sponge_mode(sponge)
    s.set_velocity_field(se.workloads.to_reference_layout(1500.0 + 1500.0 * np.random.default_rng(4).random(n)))
    rec = se.workloads.ReceiverGrid(0, 2, (nx + 1) // 2, 1, 3, (ny + 1) // 3, nz - 1)
    wav = se.workloads.ricker(30.0, dt, nt) + 1e-3
    wav[2] = np.nan  # a missing sample injects nothing

    def shot():
        seis = torch.full((nt, rec.count), 7.0, device="cuda")
        before = _launches()
        rc = se.shot_forward(s, (nx - 2, ny // 2, nz - 2), wav, nt, rec, seis=seis)  # source in the sponge
        torch.cuda.synchronize()
        return _launches() - before, rc, seis.cpu().numpy(), s.get_field(0), s.get_field(1)

    if chunks:
        monkeypatch.setenv("SEISMIC_GB300_XCHUNKS", chunks)
    shot()  # the coefficients are formed
    two = shot()
    s.set_step_fusion(1)
    one = shot()
    s.close()
    assert one[0] - two[0] == nt // 2 and one[1] == two[1]
    for a, b in zip(one[2:], two[2:]):
        assert np.abs(a).max() > 0 and np.array_equal(a, b)
