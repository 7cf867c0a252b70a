"""One SampledRays object called from several threads: traveltimes and misfits are those of the
call's own velocities, bit for bit what a single thread gets, on the device and the host path."""
import threading

import numpy as np
import pytest
import torch

import seismic_engine as se

pytestmark = pytest.mark.gpu


def test_calls_from_threads(n=24, picks=20000, threads=4, rounds=60):
    rng = np.random.default_rng(8)
    src, sta = rng.random((picks, 3)) * 1000.0, rng.random((picks, 3)) * 1000.0
    ones = np.ones(picks)
    rays = se.SampledRays((n, n, n, 50.0, 50.0, 50.0, 0.0, 0.0, 0.0), src, sta, ones, np.ones(picks, np.int8),
                          np.linalg.norm(src - sta, axis=1))
    vps = [torch.full((n ** 3,), 1000.0 * (k + 1), dtype=torch.float64, device="cuda") for k in range(threads)]
    obs = torch.zeros(picks, dtype=torch.float64, device="cuda")
    one = torch.ones(picks, dtype=torch.float64, device="cuda")
    zero = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")

    def calls(k):
        t = rays.forward_model(vps[k])
        return (t, rays.misfit(t, obs, one), rays.trial_misfit(vps[k], zero, 1.0, None, 1.0, 1e6, obs, one),
                rays.forward_model(vps[k].cpu().numpy()))

    want = [calls(k) for k in range(threads)]
    assert len({w[1] for w in want}) == threads
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(rounds):
                t, m, trial, host = calls(k)
                if not (torch.equal(t, want[k][0]) and m == want[k][1] and trial == want[k][2] and
                        np.array_equal(host, want[k][3])):
                    wrong.append(k)

    pool = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for p in pool:
        p.start()
    for p in pool:
        p.join()
    assert not wrong
