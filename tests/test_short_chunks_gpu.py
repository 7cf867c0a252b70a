"""Grids that leave multiprocessors idle are marched in the shortest x-chunks one wave of
blocks allows, down to one plane; larger ones in chunks of at most 48 planes. A chunk recomputes its halo planes with the arithmetic of
their owner, so the fields, the image and the traces are those of a single chunk bit for bit."""
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


def run(se, n, nt, fused):
    import torch
    nx, ny, nz = n
    rng = np.random.default_rng(7)
    vel = 1500.0 + 1500.0 * rng.random((nx, ny, nz))
    dt = se.workloads.cfl_dt(10.0, 3000.0)
    s = se.WaveEquationSolver(se.GridParams(nx, ny, nz, 10.0, 10.0, 10.0),
                              se.SolverConfig(dt=dt, nt=nt, sponge_width=3, sponge_damping=0.02))
    try:
        s.set_velocity_field(se.workloads.to_reference_layout(vel))
        s.set_step_fusion(fused)
        rec = se.workloads.ReceiverGrid(0, 1, nx, 0, 1, ny, nz // 2)
        data = torch.from_numpy((rng.standard_normal((nt, rec.count)) * 1e-3).astype(np.float32)).cuda()
        image, illum = (torch.zeros(nx * ny * nz, device="cuda") for _ in range(2))
        assert se.rtm_shot(s, (nx // 2, ny // 2, nz // 3), se.workloads.ricker(25.0, dt, nt), nt, rec, data, image,
                           illum, snap_kind=1) == 0
        torch.cuda.synchronize()
        return image.cpu().numpy(), illum.cpu().numpy(), s.get_field(0), s.get_field(1)
    finally:
        s.close()


# one plane; chunks of one plane (few tiles); a length that the chunks do not divide; many tiles, chunks of
# three; 52 tiles, where one wave would take longer chunks
@pytest.mark.parametrize("fused", [1, 2])
@pytest.mark.parametrize("n", [(1, 20, 24), (13, 33, 72), (31, 130, 64), (37, 100, 128), (97, 200, 256)])
def test_shortest_chunks_against_one_chunk(se, monkeypatch, n, fused):
    got = run(se, n, 13, fused)
    monkeypatch.setenv("SEISMIC_GB300_XCHUNKS", "1")
    ref = run(se, n, 13, fused)
    assert np.abs(ref[1]).max() > 0
    for a, b, what in zip(got, ref, ("image", "illumination", "current field", "previous field")):
        assert np.array_equal(a, b), what
