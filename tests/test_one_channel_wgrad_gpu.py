"""Weight gradient of the 1 to 32 layer on either side of the line between its kernels (5,000
voxels): by taps up to it, by rows beyond, the rows ragged in x, y and z. Against an FP64 sum.
Tolerance: each weight is an FP32 sum of n products, off by sqrt(n) 2^-24 in the root mean square
of random signs; 8 of these at n <= 5,418 voxels, relative to the norm of the weights alone, is
8 * 74 * 2^-24 < 4e-5."""
import numpy as np
import pytest
import torch

import seismic_engine  # noqa: F401
from seismic_engine._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(17, 17, 17), (5, 10, 100), (3, 1667, 1), (1, 9, 602), (1, 601, 9), (602, 1, 9),
                                   (5, 8, 129), (19, 17, 16), (1, 1, 5003)])
def test_either_kernel(shape):
    D, H, W = shape
    rng = np.random.default_rng(D)
    h = np.zeros((D + 2, H + 2, W + 2, 32), np.float32)
    h[1:-1, 1:-1, 1:-1] = rng.standard_normal((D, H, W, 32))
    hd = torch.from_numpy(h).bfloat16().cuda()
    dz = torch.from_numpy(rng.standard_normal((D, H, W)).astype(np.float32)).cuda()
    dw = torch.zeros(32 * 27, device="cuda")
    call("st_pc_conv1_wgrad", dz.data_ptr(), hd.data_ptr(), dw.data_ptr(), D, H, W,
         torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    hf, g = hd.cpu().double().numpy(), dz.cpu().double().numpy().reshape(-1)
    ref = np.stack([g @ hf[t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H, t % 3:t % 3 + W].reshape(-1, 32)
                    for t in range(27)], axis=1)
    got = dw.cpu().double().numpy().reshape(32, 27)
    assert np.linalg.norm(got - ref) <= 4e-5 * np.linalg.norm(ref)
