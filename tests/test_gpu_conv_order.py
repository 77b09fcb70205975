"""The order of the convolutions' sums, which is part of their results: FP32
accumulation rounds, BF16 rounding of the next layer and a training step magnify
the last bit.

Forward: an output adds its products tap by tap, t = 0 .. 26, and within a tap 16
channels at a time.  Each output channel gets three weights, +2^30, -2^30 and 1, at
three places of that order; on ones as input the 1 is lost where it comes between the
two large ones or before them (2^30 + 1 is not a float) and stays where it comes last, so
the output tells the order.

Weight gradient: accumulation in tensor memory rounds towards zero, so the error of a
sum of positive terms grows with the number n of MMAs in a chain.  In the mean each
loses half a unit in the last place by the rounding and as much by aligning what it
adds, of partial sums that are half of the whole; a unit is at most 2^-23 of its number:
n 2^-24.  n is that of an equal share of the 128-voxel tiles per multiprocessor; the FP32
sums of the shares add 2^-23."""
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


@pytest.mark.parametrize("shape,cin,cout", [((52, 32, 128), 48, 16), ((28, 32, 64), 96, 32), ((92, 32, 64), 32, 32),
                                            ((44, 16, 128), 64, 64), ((13, 16, 32), 64, 32)])
def test_weight_gradient_chains(ctx, shape, cin, cout):  # noqa: F811
    import torch
    D, H, W = shape
    g = torch.Generator(device="cuda").manual_seed(cin + D)
    x = torch.rand(D, H, W, cin, device="cuda", generator=g).bfloat16()
    dy = torch.rand(D, H, W, cout, device="cuda", generator=g).bfloat16()
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    v = dy.double().reshape(-1, cout).T
    want = torch.stack([v @ xp[t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H, t % 3:t % 3 + W].reshape(-1, cin)
                        for t in range(27)])
    dw = torch.zeros(27, cout, cin, device="cuda")
    torch.cuda.synchronize()
    d = A.ConvDesc(D, H, W, cin, cout, 0)
    A.cuda_check(ctx.lib.artss_conv3d_wgrad(ctx.h, C.byref(d), x.data_ptr(), dy.data_ptr(), dw.data_ptr()), "wgrad")
    A.cuda_check(ctx.lib.artss_nn_check(ctx.h), "wait")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 8 * -(-D * H * W // 128 // sms)
    off = float((dw.double() / want - 1).abs().mean())
    assert off <= n * 2.0 ** -24 + 2.0 ** -23, (off, n)
