"""Tile edges of the tensor-core convolutions: grids narrower and flatter than a
block's 8 x 16 voxels, depths that leave a part of the block's planes, and channel
counts that split over blocks, against the FP32 numpy convolutions of the same
BF16 inputs (tolerances as in test_gpu_conv.py: BF16 rounding of the output, FP32
accumulation order of the gradient)."""
import ctypes as C

import numpy as np
import pytest

import artss_b200 as A
from artss_b200 import learned as LN
from tests.test_gpu_conv import ctx, dev_bf16  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,cin,cout", [((8, 4, 4), 16, 16), ((1, 128, 1), 16, 48), ((17, 4, 32), 32, 16),
                                            ((3, 24, 16), 16, 112), ((5, 8, 64), 64, 128), ((2, 1, 128), 112, 16)])
def test_forward_and_weight_gradient(ctx, shape, cin, cout):  # noqa: F811
    import torch
    D, H, W = shape
    rng = np.random.default_rng(cin + 3 * cout + D)
    x = LN.round_bf16(rng.standard_normal((D, H, W, cin)).astype(np.float32))
    w = LN.round_bf16((rng.standard_normal((cout, cin, 3, 3, 3)) / np.sqrt(27 * cin)).astype(np.float32))
    bias = rng.standard_normal(cout).astype(np.float32)
    g = LN.round_bf16(rng.standard_normal((D, H, W, cout)).astype(np.float32))
    dx, dwp, dg, db = dev_bf16(x), dev_bf16(LN.pack_conv_weights(w)), dev_bf16(g), torch.from_numpy(bias).cuda()
    dy = torch.full((D * H * W * cout + 64,), 7.0, dtype=torch.bfloat16, device="cuda")
    dw = torch.zeros((27, cout, cin), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    d = A.ConvDesc(D, H, W, cin, cout, 0)
    A.cuda_check(ctx.lib.artss_conv3d_fwd(ctx.h, C.byref(d), dx.data_ptr(), dwp.data_ptr(), db.data_ptr(), dy.data_ptr()),
                 "conv")
    A.cuda_check(ctx.lib.artss_conv3d_wgrad(ctx.h, C.byref(d), dx.data_ptr(), dg.data_ptr(), dw.data_ptr()), "wgrad")
    A.cuda_check(ctx.lib.artss_nn_check(ctx.h), "wait")
    got = dy.float().cpu().numpy()
    assert (got[-64:] == 7.0).all()
    ref = LN.conv3d_ref(x, w, bias)
    assert np.abs(got[:-64].reshape(ref.shape) - ref).max() <= 1e-2 * np.abs(ref).max()
    ref = LN.conv3d_wgrad_ref(x, g)
    assert np.abs(dw.cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max() + 1e-4


def test_refused_operands(ctx):  # noqa: F811
    """what the operands' size ruled out is still refused"""
    import torch
    t = torch.zeros(1 << 16, dtype=torch.bfloat16, device="cuda")
    d = A.ConvDesc(1, 1, 128, 256, 256, 0)
    assert ctx.lib.artss_conv3d_fwd(ctx.h, C.byref(d), t.data_ptr(), t.data_ptr(), None, t.data_ptr()) == -6
    d = A.ConvDesc(1, 3, 100, 16, 16, 0)
    assert ctx.lib.artss_conv3d_fwd(ctx.h, C.byref(d), t.data_ptr(), t.data_ptr(), None, t.data_ptr()) == -1
