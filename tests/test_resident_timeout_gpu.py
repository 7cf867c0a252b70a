"""The bounded waits of the resident shot, without a GPU fault: the first block leaves before
the first step, so its neighbours' waits run out after 1 ms, every block leaves and the call returns
ST_ERR_TIMEOUT. The next shot of the same handle gives what one step per launch gives, bit for bit.
One, two, four and eight planes per block, both sponge rules."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine._lib import ST_ERR_TIMEOUT, call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sponge", ["reference", "stable"])
@pytest.mark.parametrize("n", [(24, 24, 24), (48, 40, 56), (64, 64, 64), (112, 112, 112), (20, 20, 1000)])
def test_a_lost_block_times_out_and_the_handle_recovers(n, sponge):
    nt = 10
    dt = se.workloads.cfl_dt(10.0, 3000.0)
    s = se.WaveEquationSolver(se.GridParams(*n, 10.0, 10.0, 10.0),
                              se.SolverConfig(dt=dt, nt=nt, sponge_width=4, sponge_damping=0.02))
    s.set_sponge_mode(sponge)
    s.set_velocity_field(se.workloads.to_reference_layout(1500.0 + 1500.0 * np.random.default_rng(2).random(n)))
    rec = se.workloads.ReceiverGrid(0, 1, n[0], 0, 1, n[1], 5)
    wav = se.workloads.ricker(30.0, dt, nt) + 1e-3

    def shot():
        seis = torch.zeros((nt, rec.count), device="cuda")
        se.shot_forward(s, (n[0] // 2, n[1] // 2, 6), wav, nt, rec, seis=seis)
        torch.cuda.synchronize()
        return seis.cpu().numpy(), s.get_field(0), s.get_field(1)

    s.set_step_fusion(1)
    one = shot()
    s.set_step_fusion(2)
    for _ in range(2):
        call("st_solver_set_wait_test", s.handle, 1_000_000, -2)
        with pytest.raises(se.SeismicError) as e:
            shot()
        assert e.value.code == ST_ERR_TIMEOUT
        call("st_solver_set_wait_test", s.handle, 0, -1)
        for a, b in zip(one, shot()):
            assert np.array_equal(a, b)
    assert np.abs(one[0]).max() > 0
    s.close()
