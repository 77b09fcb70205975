"""The network's element-wise kernels one by one, in the form that moves 8 channels at a
time and in the one for odd channel counts and unaligned arrays: exactly the values of
the same BF16 / FP32 operations in torch, sums within their order's rounding."""
import ctypes as C

import pytest

import artss_b200 as A
from tests.test_gpu_conv import ctx  # noqa: F401

pytestmark = pytest.mark.gpu
# channels, offset of the arrays in elements (8 elements are 16 bytes)
FORMS = [(8, 0), (48, 0), (16, 3), (7, 0), (1, 1), (12, 0)]


def P(t):
    return C.c_void_p(t.data_ptr())


class Arrays:
    """BF16 arrays `off` elements behind an aligned address, with guard elements around"""

    def __init__(self, seed, off):
        import torch
        self.torch, self.off, self.bases = torch, off, []
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, n, fill=None):
        base = self.torch.full((n + 32,), 7.0, dtype=self.torch.bfloat16, device="cuda")
        v = base[8 + self.off:8 + self.off + n]
        v.copy_(self.torch.randn(n, device="cuda", generator=self.g) if fill is None else
                self.torch.full((n,), fill, device="cuda"))
        self.bases.append((base, n))
        return v

    def run(self, ctx, st, what):  # noqa: F811
        A.cuda_check(st, what)
        A.cuda_check(ctx.lib.artss_nn_check(ctx.h), what)
        for base, n in self.bases:
            assert bool((base[:8 + self.off] == 7.0).all()) and bool((base[8 + self.off + n:] == 7.0).all())


def same(got, want):
    import torch
    return torch.equal(got.reshape(-1), want.reshape(-1).to(got.dtype))


@pytest.mark.parametrize("c,off", FORMS)
def test_relu_backward(ctx, c, off):  # noqa: F811
    import torch
    new = Arrays(c, off)
    n = 1003 * c
    dy, y = new(n), new(n)
    y[::5] = 0.0
    want = torch.where(y > 0, dy, torch.zeros_like(dy))
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_relu_bwd(ctx.h, P(dy), P(y), C.c_int64(n)), "relu")
    assert same(dy, want)


@pytest.mark.parametrize("c,off", FORMS)
def test_pool(ctx, c, off):  # noqa: F811
    import torch
    D, H, W = 6, 4, 10
    new = Arrays(c, off)
    x, y = new(D * H * W * c), new(D * H * W // 8 * c, 0.0)
    v = x.float().reshape(D // 2, 2, H // 2, 2, W // 2, 2, c)
    s = torch.zeros(D // 2, H // 2, W // 2, c, device="cuda")
    for o in range(8):
        s = s + v[:, o >> 2, :, o >> 1 & 1, :, o & 1]
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_pool2(ctx.h, P(x), P(y), D, H, W, c, 0), "pool")
    assert same(y, 0.125 * s)
    dy, dx = new(D * H * W // 8 * c), new(D * H * W * c, 0.0)
    want = (0.125 * dy.float()).reshape(D // 2, 1, H // 2, 1, W // 2, 1, c).expand(-1, 2, -1, 2, -1, 2, -1)
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_pool2(ctx.h, P(dy), P(dx), D, H, W, c, 1), "pool backward")
    assert same(dx, want)


@pytest.mark.parametrize("c,off", FORMS)
@pytest.mark.parametrize("c_off", [0, 8, 3])
def test_upsampling(ctx, c, off, c_off):  # noqa: F811
    import torch
    D, H, W = 3, 2, 5
    total = c + c_off + (8 if c % 8 == 0 else 2)
    new = Arrays(c, off)
    x, y = new(D * H * W * c), new(8 * D * H * W * total)
    want = y.clone().reshape(D, 2, H, 2, W, 2, total)
    want[..., c_off:c_off + c] = x.reshape(D, 1, H, 1, W, 1, c)
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_up2(ctx.h, P(x), P(y), D, H, W, c, total, c_off, 0), "up")
    assert same(y, want)
    dy, dx = new(8 * D * H * W * total), new(D * H * W * c, 0.0)
    v = dy.float().reshape(D, 2, H, 2, W, 2, total)[..., c_off:c_off + c]
    s = torch.zeros(D, H, W, c, device="cuda")
    for o in range(8):
        s = s + v[:, o >> 2, :, o >> 1 & 1, :, o & 1]
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_up2(ctx.h, P(dy), P(dx), D, H, W, c, total, c_off, 1), "up backward")
    assert same(dx, s)


@pytest.mark.parametrize("c,off", FORMS)
@pytest.mark.parametrize("s_off,d_off,accumulate", [(0, 0, 0), (8, 16, 1), (1, 0, 1), (0, 5, 0)])
def test_copy_channels(ctx, c, off, s_off, d_off, accumulate):  # noqa: F811
    import torch
    voxels, s_total, d_total = 777, c + s_off + 8, c + d_off
    new = Arrays(c, off)
    src, dst = new(voxels * s_total), new(voxels * d_total)
    s, want = src.reshape(voxels, s_total)[:, s_off:s_off + c], dst.clone().reshape(voxels, d_total)
    old = want[:, d_off:d_off + c]
    want[:, d_off:d_off + c] = (old.float() + s.float()).bfloat16() if accumulate else s
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_copy_channels(ctx.h, P(src), s_total, s_off, P(dst), d_total, d_off, c, C.c_int64(voxels),
                                                accumulate), "copy")
    assert same(dst, want)


@pytest.mark.parametrize("c,off", [(16, 0), (8, 0), (16, 1), (3, 0)])
def test_loss_gradient(ctx, c, off):  # noqa: F811
    """the loss is a sum of 1003 FP32 terms: 2^-20 of it"""
    import torch
    voxels, inv = 1003, 1.0 / 900.0
    new = Arrays(c, off)
    y, dy, mask = new(voxels * c), new(voxels * c, 0.0), new(voxels * c)
    t = torch.randn(voxels, device="cuda", generator=new.g)
    part = torch.empty(5, device="cuda")
    inside = mask.reshape(voxels, c)[:, 1].float() > 0.5
    d = torch.where(inside, y.reshape(voxels, c)[:, 0].float() - t, torch.zeros_like(t))
    want = torch.zeros(voxels, c, device="cuda")
    want[:, 0] = d * torch.tensor(inv, dtype=torch.float32)
    torch.cuda.synchronize()
    new.run(ctx, ctx.lib.artss_nn_mse(ctx.h, P(y), c, P(t), P(mask), P(dy), C.c_int64(voxels), C.c_float(inv), P(part), 5),
            "loss")
    assert same(dy, want)
    loss = float((0.5 * d.double() ** 2).sum())
    assert abs(float(part.double().sum()) - loss) <= 2.0 ** -20 * loss


@pytest.mark.parametrize("voxels,c", [(28 * 32 * 64, 32), (11 * 16 * 32, 64), (52 * 64 * 128, 16), (1001, 96), (1, 8), (0, 8),
                                      (777, 7), (513, 300), (5, 1)])
def test_bias_gradient(ctx, voxels, c):  # noqa: F811
    """added to what the array holds; chains of a few hundred FP32 additions with independent roundings: 2^-20 of
    the sum of absolute values"""
    import torch
    g = torch.Generator(device="cuda").manual_seed(c)
    dy = torch.randn(max(voxels, 1) * c, device="cuda", generator=g).bfloat16()
    v = dy[:voxels * c].double().reshape(voxels, c)
    db = torch.full((c,), 3.0, device="cuda")
    torch.cuda.synchronize()
    A.cuda_check(ctx.lib.artss_nn_bias_grad(ctx.h, C.c_void_p(dy.data_ptr()), C.c_void_p(db.data_ptr()), C.c_int64(voxels), c),
                 "bias")
    A.cuda_check(ctx.lib.artss_nn_check(ctx.h), "wait")
    assert bool(((db.double() - 3.0 - v.sum(0)).abs() <= 2.0 ** -20 * (3.0 + v.abs().sum(0))).all())
