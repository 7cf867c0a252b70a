"""Forward shots whose grid stays on the SMs for all steps, against one launch per step: the
same arithmetic in the same order, so seismograms and fields are bit-identical. The shapes take
every number of planes per block, blocks that the grid fills in part in x, y and z, one row and
one column per block, a single block, and a grid that does not fit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def se():
    import importlib.util
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    spec = importlib.util.spec_from_file_location(
        "st_build", os.path.join(repo, "03-seismic-tomography-compute_gb300", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    mod.build()
    import seismic_engine
    return seismic_engine


def solver(se, n, nt, sponge):
    nx, ny, nz = n
    vel = 1500.0 + 1500.0 * np.random.default_rng(11).random((nx, ny, nz))
    dt = se.workloads.cfl_dt(10.0, 3000.0)
    s = se.WaveEquationSolver(se.GridParams(nx, ny, nz, 10.0, 10.0, 10.0),
                              se.SolverConfig(dt=dt, nt=nt, sponge_width=4, sponge_damping=0.02))
    s.set_sponge_mode(sponge)
    s.set_velocity_field(se.workloads.to_reference_layout(vel))
    return s


def shot(se, s, n, nt, src, wav, rec):
    import torch
    seis = torch.full((nt, rec.count), 7.0, device="cuda")
    rc = se.shot_forward(s, src, wav, nt, rec, seis=seis)
    torch.cuda.synchronize()
    return rc, seis.cpu().numpy(), s.get_field(0), s.get_field(1)


def compare(one, two):
    assert one[0] == two[0]
    for a, b, what in zip(one[1:], two[1:], ("seismograms", "current field", "previous field")):
        assert np.array_equal(a, b), what


CASES = [
    # (nx, ny, nz), nt, sponge rule, source
    ((1, 1, 1), 9, "reference", (0, 0, 0)),
    ((3, 3, 3), 8, "reference", (1, 1, 1)),         # one column per block
    ((9, 40, 17), 21, "stable", (8, 3, 16)),        # nz % 4 = 1, source on the last x and z, last row of a block
    ((48, 40, 56), 64, "reference", (24, 21, 28)),  # two planes, source on a block's first row and plane
    ((300, 5, 5), 15, "stable", (149, 2, 4)),       # one block in y
    ((20, 11, 2047), 12, "reference", (3, 5, 127)),  # one row per block, the halo rows in several rounds
    ((33, 18, 700), 16, "stable", (32, 17, 128)),   # four planes, the last block one plane
    ((121, 127, 126), 33, "reference", (56, 45, 3)),  # eight planes, all three extents ragged
    ((160, 160, 160), 9, "reference", (80, 80, 80)),  # does not fit
]


@pytest.mark.parametrize("n,nt,sponge,src", CASES)
def test_resident_shot_bit_identical(se, n, nt, sponge, src):
    nx, ny, nz = n
    dt = se.workloads.cfl_dt(10.0, 3000.0)
    rec = se.workloads.ReceiverGrid(0, 3, (nx + 2) // 3, 0, 2, (ny + 1) // 2, nz // 2)
    s = solver(se, n, nt, sponge)
    try:
        # a missing sample injects nothing
        wav = se.workloads.ricker(30.0, dt, nt) + 1e-3
        wav[3] = np.nan
        s.set_step_fusion(1)
        one = shot(se, s, n, nt, src, wav, rec)
        s.set_step_fusion(2)
        for _ in range(2):  # a second launch goes on with the tags of the first
            compare(one, shot(se, s, n, nt, src, wav, rec))
        assert np.abs(one[2]).max() > 0
    finally:
        s.close()


def test_resident_shot_clamps_alike(se):
    n, nt = (24, 30, 44), 20
    rec = se.workloads.ReceiverGrid(0, 1, 24, 0, 1, 30, 20)
    s = solver(se, n, nt, "reference")
    try:
        wav = np.zeros(nt)
        wav[0], wav[4] = 1e12, 3e38  # past the amplitude limit, then out of range
        s.set_step_fusion(1)
        one = shot(se, s, n, nt, (12, 9, 20), wav, rec)
        s.set_step_fusion(2)
        compare(one, shot(se, s, n, nt, (12, 9, 20), wav, rec))
    finally:
        s.close()


@pytest.mark.parametrize("nt", [8, 21])
def test_resident_shot_leaves_the_third_field_alike(se, monkeypatch, nt):
    n = (24, 30, 44)
    rec = se.workloads.ReceiverGrid(0, 1, 24, 0, 1, 30, 20)
    s = solver(se, n, nt, "reference")
    try:
        wav = se.workloads.ricker(30.0, se.workloads.cfl_dt(10.0, 3000.0), nt) + 1e-3
        got = shot(se, s, n, nt, (12, 9, 20), wav, rec) + (s.get_field(2),)
        monkeypatch.setenv("SEISMIC_GB300_XCHUNKS", "3")  # launches of two steps
        want = shot(se, s, n, nt, (12, 9, 20), wav, rec) + (s.get_field(2),)
        compare(want, got)
        assert np.abs(want[4]).max() > 0 and np.array_equal(want[4], got[4])
    finally:
        s.close()


def test_resident_shots_from_two_streams(se):
    import threading
    n, nt = (48, 40, 56), 100
    rec = se.workloads.ReceiverGrid(0, 1, 48, 0, 1, 40, 20)
    wav = se.workloads.ricker(30.0, se.workloads.cfl_dt(10.0, 3000.0), nt)
    solvers = [solver(se, n, nt, "reference") for _ in range(3)]
    try:
        want = shot(se, solvers[0], n, nt, (24, 20, 28), wav, rec)
        got = [[] for _ in solvers]

        def work(i):
            for _ in range(4):
                got[i].append(shot(se, solvers[i], n, nt, (24, 20, 28), wav, rec))

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(solvers))]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        for results in got:
            assert len(results) == 4
            for r in results:
                compare(want, r)
    finally:
        for s in solvers:
            s.close()
