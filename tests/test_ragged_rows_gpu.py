"""Two steps per launch on rows that are not multiples of 16 bytes: the padded
library-owned store against one step per launch and against a caller's compact
store, bit for bit (images, illumination, reflectivity, seismograms, fields)."""
import numpy as np
import pytest
import torch

import seismic_engine as se
from seismic_engine import _lib

pytestmark = pytest.mark.gpu
KINDS = {"bf16": (_lib.ST_SNAP_BF16, torch.bfloat16), "fp16": (_lib.ST_SNAP_FP16, torch.float16),
         "fp32": (_lib.ST_SNAP_FP32, torch.float32)}


def _solver(w, fused):
    s = se.WaveEquationSolver(se.GridParams(w.nx, w.ny, w.nz, w.d, w.d, w.d),
                              se.SolverConfig(dt=w.dt, nt=w.nt, sponge_width=w.sponge_width,
                                              sponge_mode=w.sponge_mode))
    s.set_velocity_field(se.workloads.to_reference_layout(w.vel))
    s.set_step_fusion(fused)
    return s


@pytest.mark.parametrize("mode", ["stable", "reference"])
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("shape,nt", [((9, 18, 5), 13), ((20, 17, 65), 14), ((14, 33, 67), 9), ((12, 16, 100), 10),
                                      ((5, 6, 30), 2)])
def test_padded_store(shape, nt, kind, mode):
    w = se.workloads.small_case(n=shape, nt=nt, sponge_width=2)
    w.sponge_mode = mode
    sh = w.shots[0]
    sk, dt = KINDS[kind]
    n = w.points
    data = torch.randn((nt, sh.rec.count), generator=torch.Generator().manual_seed(nt)).cuda()
    out = []
    for fused, own in ((2, True), (1, True), (2, False)):
        s = _solver(w, fused)
        snaps = None if own else torch.zeros((nt, n), dtype=dt, device="cuda")
        amax = None if own else torch.zeros(nt + 1, dtype=torch.int32, device="cuda")
        im = [torch.full((n,), 3.0, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        se.rtm_shot(s, sh.src, sh.wavelet, nt, sh.rec, data, *im, snap_kind=sk, snaps=snaps, snap_amax=amax)
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in im])
        if own:  # the host entry point takes the same store
            got = se.rtm_shot_host(s, None, sh.src, sh.wavelet, nt, sh.rec, data.cpu(), snap_kind=sk)
            for a, b in zip(out[-1], (got["image"], got["illumination"], got["reflectivity"])):
                np.testing.assert_array_equal(a, b.astype(np.float32))
        s.close()
    assert np.abs(out[0][1]).max() > 0  # two steps carry no data to the source: no image yet, but illumination
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("shape,nt", [((9, 18, 1), 8), ((7, 40, 63), 11), ((30, 5, 66), 12), ((16, 16, 131), 7)])
def test_forward_pairs(shape, nt):
    w = se.workloads.small_case(n=shape, nt=nt, sponge_width=2) if shape[2] > 4 else None
    if w is None:
        w = se.workloads.small_case(n=(shape[0], shape[1], 28), nt=nt, sponge_width=2)
        w.nz, w.vel = shape[2], np.ascontiguousarray(w.vel[:, :, :shape[2]])
        w.shots[0].src = (shape[0] // 2, shape[1] // 2, 0)
        w.shots[0].rec.z = 0
    sh = w.shots[0]
    res = []
    for fused in (2, 1):
        s = _solver(w, fused)
        seis = torch.zeros((nt, sh.rec.count), device="cuda")
        torch.cuda.synchronize()
        se.shot_forward(s, sh.src, sh.wavelet, nt, sh.rec, seis=seis)
        torch.cuda.synchronize()
        res.append((seis.cpu().numpy(), s.get_field(0), s.get_field(1)))
        s.close()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)
    assert np.abs(res[0][1]).max() > 0
