"""The order of the convolutions' sums, which is part of their results: FP32
accumulation rounds, BF16 rounding of the next layer and a training step magnify
the last bit.

Forward: an output adds its products tap by tap, t = 0 .. 26, and within a tap 16
channels at a time.  Each output channel gets three weights, +2^30, -2^30 and 1, at
three places of that order; on ones as input the 1 is lost where it comes between the
two large ones or before them (2^30 + 1 is not a float) and stays where it comes last, so
the output tells the order."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import learned as LN
from tests.test_gpu_conv import ctx, dev_bf16  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,cin,cout", [((5, 16, 32), 16, 16), ((12, 16, 64), 48, 16), ((9, 16, 32), 96, 32),
                                            ((7, 16, 16), 64, 64), ((3, 24, 16), 32, 96), ((17, 4, 32), 80, 32),
                                            ((4, 8, 16), 256, 80), ((33, 16, 32), 112, 48)])
def test_forward_adds_tap_by_tap(ctx, shape, cin, cout):  # noqa: F811
    import torch
    D, H, W = shape
    rng = np.random.default_rng(cin + cout + D)
    w = np.zeros((27, cout, cin), np.float32)
    want = np.zeros(cout, np.float32)
    for co in range(cout):
        place = rng.choice(27 * (cin // 16), 3, replace=False)  # tap * groups of 16 channels + group
        for value, p in zip((2.0 ** 30, -2.0 ** 30, 1.0), place):
            w[p // (cin // 16), co, 16 * (p % (cin // 16)) + rng.integers(16)] = value
        want[co] = float(place[2] == max(place))
    assert 0 < want.sum() < cout
    wp = w.reshape(27, cout, cin // 8, 8).transpose(0, 2, 1, 3)  # [tap][C_in / 8][C_out][8]
    x, dwp = dev_bf16(np.ones((D, H, W, cin), np.float32)), dev_bf16(np.ascontiguousarray(wp))
    y = torch.empty(D * H * W * cout, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    d = A.ConvDesc(D, H, W, cin, cout, 0)
    A.cuda_check(ctx.lib.artss_conv3d_fwd(ctx.h, C.byref(d), x.data_ptr(), dwp.data_ptr(), None, y.data_ptr()), "conv")
    A.cuda_check(ctx.lib.artss_nn_check(ctx.h), "wait")
    inside = y.float().cpu().numpy().reshape(D, H, W, cout)[1:-1, 1:-1, 1:-1]  # every tap reads a voxel
    assert (inside == want).all()
