"""Weight gradient of the 32 -> 32 layer at the edges of its tiling: volumes of less than one
K step (128 padded rows), one step more than the blocks share evenly, rows shorter and longer
than a step; accumulation into a non-zero dW. Against an FP64 sum over the interior voxels.
Tolerance: each weight is an FP32 sum of n products of BF16 values (exact in FP32), in partial
sums; n 2^-24 in the worst case, and sqrt(n) 2^-24 <= 3e-5 in the root mean square of random
signs at the largest n here (57,000 voxels): relative to the norm, 3e-5 bounds both."""
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


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (1, 2, 40), (14, 14, 6), (3, 4, 300), (32, 32, 32), (30, 38, 50)])
def test_wgrad_edges(se, shape):
    import torch
    from seismic_engine._lib import call
    st = torch.cuda.current_stream().cuda_stream
    D, H, W = shape
    gen = torch.Generator().manual_seed(sum(shape))
    x = torch.zeros((D + 2, H + 2, W + 2, 32))
    x[1:-1, 1:-1, 1:-1] = torch.randn((D, H, W, 32), generator=gen)
    xb = x.bfloat16()
    gb = torch.randn((D + 2, H + 2, W + 2, 32), generator=gen).bfloat16()  # the border rows count for nothing
    start = torch.randn(32 * 32 * 27, generator=gen)
    dw = start.cuda()
    xd, gd = xb.cuda(), gb.cuda()
    call("st_conv3d_wgrad", xd.data_ptr(), gd.data_ptr(), dw.data_ptr(), D, H, W, st)
    call("st_conv3d_check", st)
    xf, gi = xb.double().numpy(), gb.double().numpy()[1:-1, 1:-1, 1:-1].reshape(-1, 32)
    ref = np.zeros((32, 32, 27))
    for tap in range(27):
        kd, kh, kw = tap // 9, (tap // 3) % 3, tap % 3
        ref[:, :, tap] = gi.T @ xf[kd:kd + D, kh:kh + H, kw:kw + W].reshape(-1, 32)
    ref += start.double().numpy().reshape(32, 32, 27)
    got = dw.cpu().double().numpy().reshape(32, 32, 27)
    assert np.linalg.norm(got - ref) <= 3e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 9, 8), (5, 8, 9), (3, 17, 33), (32, 32, 32), (2, 7, 300)])
def test_one_channel_wgrad_edges(se, shape):
    import torch
    from seismic_engine._lib import call
    st = torch.cuda.current_stream().cuda_stream
    D, H, W = shape
    gen = torch.Generator().manual_seed(sum(shape))
    h = torch.zeros((D + 2, H + 2, W + 2, 32))
    h[1:-1, 1:-1, 1:-1] = torch.randn((D, H, W, 32), generator=gen)
    hb = h.bfloat16()
    dz = torch.randn((D, H, W), generator=gen)
    start = torch.randn(32 * 27, generator=gen)
    dw, dzd, hd = start.cuda(), dz.cuda(), hb.cuda()
    call("st_pc_conv1_wgrad", dzd.data_ptr(), hd.data_ptr(), dw.data_ptr(), D, H, W, st)
    torch.cuda.synchronize()
    hf, g = hb.double().numpy(), dz.double().numpy().reshape(-1)
    ref = start.double().numpy().reshape(32, 27).copy()
    for tap in range(27):
        kd, kh, kw = tap // 9, (tap // 3) % 3, tap % 3
        ref[:, tap] += g @ hf[kd:kd + D, kh:kh + H, kw:kw + W].reshape(-1, 32)
    got = dw.cpu().double().numpy().reshape(32, 27)
    assert np.linalg.norm(got - ref) <= 3e-5 * np.linalg.norm(ref)
