"""The convolution's tile choices at their edges against FP64 conv3d of the same
BF16 values (relative L2 <= 1e-5: FP32 accumulation of 864 exact products):
single voxels and planes, tiles of 128 and 256 voxels, one to three window
slots, several rounds of units; and that a non-finite voxel reaches its 3 x 3 x 3
neighbourhood and no further (a plane's lanes are shared with the planes four
away)."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

from test_conv_gpu import lib, pack, padded, rel, run_conv, unpad  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,H,W", [(1, 1, 1), (1, 40, 40), (2, 1, 126), (9, 130, 110), (6, 60, 229), (3, 50, 230),
                                   (2, 3, 268), (40, 12, 14), (11, 200, 63)])
def test_tiles(lib, D, H, W):  # noqa: F811
    g = torch.Generator().manual_seed(D + H + W)
    x = torch.randn((32, D, H, W), generator=g)
    w = (torch.randn((32, 32, 3, 3, 3), generator=g) / 30).cuda()
    xin = padded(x)
    out = run_conv(lib, xin, pack(lib, w), None, xin, D, H, W, relu=False, f32=True)
    xb = xin[1:-1, 1:-1, 1:-1].permute(3, 0, 1, 2).double()
    ref = F.conv3d(xb[None].cpu(), w.to(torch.bfloat16).double().cpu(), padding=1)[0] + xb.cpu()
    assert rel(unpad(out), ref) < 1e-5
    border = out.clone()
    border[1:-1, 1:-1, 1:-1] = 0
    assert not border.any()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_bad_voxel_stays_in_its_neighbourhood(lib, bad):  # noqa: F811
    D, H, W = 23, 19, 21
    x = torch.randn((32, D, H, W), generator=torch.Generator().manual_seed(1))
    w = (torch.randn((32, 32, 3, 3, 3), generator=torch.Generator().manual_seed(2)) / 30).cuda()
    clean = run_conv(lib, padded(x), pack(lib, w), None, None, D, H, W, relu=False, f32=True)
    x[:, 11, 7, 9] = bad
    out = run_conv(lib, padded(x), pack(lib, w), None, None, D, H, W, relu=False, f32=True)
    near = np.zeros((D + 2, H + 2, W + 2), bool)
    near[11:14, 7:10, 9:12] = True
    a, b = out.cpu().numpy(), clean.cpu().numpy()
    np.testing.assert_array_equal(a[~near], b[~near])
    assert not np.isfinite(a[near]).all(axis=-1).any()
