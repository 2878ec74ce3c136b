"""GPU tests of the implicit-GEMM 3x3 convolution (ds_conv3x3_*) at the edges of
its tiles: one pixel, rows and columns that fill no tile, several images in a
tile, channel counts below and above a column tile.

The forward equals im2col + GEMM bit for bit (the same products in the same
order).  Gradients are compared with FP64: dx is stored as BF16 (2^-9 relative,
held to 4e-3 in the norm); gw is summed in FP32 in chains of at most 4096
pixels, 256 tensor-core steps that may each lose 2^-23 of the running sum, so
3.1e-5 of the partial sums, held to 1e-4 of the result's norm."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [  # batch, height, width, cin, cout
    (8, 1, 1, 64, 8), (8, 1, 9, 32, 64), (16, 3, 2, 64, 56), (8, 17, 23, 32, 32),
    (8, 16, 16, 64, 128), (8, 31, 33, 128, 64), (8, 9, 130, 64, 64), (8, 5, 4, 192, 320),
    (16, 8, 8, 320, 264), (1, 64, 200, 256, 256)]


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("B,H,W,cin,cout", SHAPES)
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("act", [True, False])
def test_conv_matches_im2col_and_fp64(cuda_lib, B, H, W, cin, cout, stride, act):
    import torch
    import torch.nn.functional as F
    from diffsplat_b200 import nn
    gen = torch.Generator().manual_seed(cin + cout + H)
    conv = nn.Conv3x3(cin, cout, stride, gelu=act, gen=gen)
    conv.b.copy_(torch.randn(cout, generator=gen))
    x = torch.randn(B, H, W, cin, generator=gen).to(torch.bfloat16).cuda()
    zprev = torch.randn(B, H, W, cin, generator=gen).to(torch.bfloat16).cuda()
    gemm = nn.Gemm()
    got = conv.forward(gemm, x)
    assert conv.col is None  # the implicit path ran
    col, _ = nn.im2col(x, stride, conv.kp)
    if act:
        z, y = gemm(col, conv.w16, nn.EPI_BIAS_GELU, bias=conv.b)
        assert torch.equal(got[0].view(z.shape), z) and torch.equal(got[1].view(y.shape), y)
    else:
        assert torch.equal(got[0].view(-1, cout), gemm(col, conv.w16, nn.EPI_BIAS_F32,
                                                       bias=conv.b))
    x.fill_(float("nan"))  # the backward works on the input as the forward saw it
    dz = torch.randn(got[0].shape, generator=gen).to(torch.bfloat16).cuda()
    if dz.numel() // cout % 8:
        with pytest.raises(RuntimeError):
            conv.backward(gemm, dz, z_prev=zprev)
        return
    dx = conv.backward(gemm, dz, z_prev=zprev)
    plain = conv.backward(gemm, dz)
    torch.cuda.synchronize()
    gemm.check()
    xr = conv.x.double().permute(0, 3, 1, 2).requires_grad_(True)
    w4 = conv.w16.double()[:, :9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
    wr = w4.contiguous().requires_grad_(True)
    out = F.conv2d(xr, wr, stride=stride, padding=1)
    gx, gw = torch.autograd.grad(out, (xr, wr), dz.double().permute(0, 3, 1, 2))
    assert _rel(conv.gw[:, :9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2), gw) < 1e-4
    assert (conv.gw[:, 9 * cin:] == 0).all()
    assert _rel(conv.gb, dz.double().sum((0, 1, 2))) < 1e-5
    gx = gx.permute(0, 2, 3, 1)
    assert _rel(plain, gx) < 4e-3
    zp = zprev.double().requires_grad_(True)
    slope = torch.autograd.grad(F.gelu(zp, approximate="tanh").sum(), zp)[0]
    assert _rel(dx, gx * slope) < 4e-3


@pytest.mark.parametrize("B,H,W,cout", [(1, 1, 1, 8), (3, 7, 5, 32), (2, 40, 33, 56),
                                        (1, 130, 300, 72), (64, 9, 9, 32)])
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("act", [True, False])
def test_rgb_layer_equals_im2col(cuda_lib, B, H, W, cout, stride, act):
    import torch
    from diffsplat_b200 import nn
    gen = torch.Generator().manual_seed(cout + H)
    conv = nn.Conv3x3(3, cout, stride, gelu=act, gen=gen)
    conv.b.copy_(torch.randn(cout, generator=gen))
    x = torch.randn(B, H, W, 3, generator=gen).to(torch.bfloat16).cuda()
    gemm = nn.Gemm()
    got = conv.forward(gemm, x)
    assert conv.col is None
    col, _ = nn.im2col(x, stride, conv.kp)
    torch.cuda.synchronize()
    gemm.check()
    if act:
        z, y = gemm(col, conv.w16, nn.EPI_BIAS_GELU, bias=conv.b)
        assert torch.equal(got[0].view(z.shape), z) and torch.equal(got[1].view(y.shape), y)
    else:
        d = gemm(col, conv.w16, nn.EPI_BIAS_F32, bias=conv.b)
        assert torch.equal(got[0].view(-1, cout), d)


def test_conv_timeout_is_reported_and_device_stays_usable(cuda_lib):
    """Pipeline waits limited to one poll: the waits run out, what was issued
    lands, TMEM is freed and the error word is set; then a normal call works."""
    import torch
    from diffsplat_b200 import nn
    conv = nn.Conv3x3(64, 64, 1, gen=torch.Generator().manual_seed(0))
    x = torch.randn(4, 64, 64, 64).to(torch.bfloat16).cuda()
    gemm = nn.Gemm()
    z0, _ = conv.forward(gemm, x)
    torch.cuda.synchronize()
    nn.set_spin_limit(1)
    try:
        conv.forward(gemm, x)
        torch.cuda.synchronize()
    finally:
        nn.set_spin_limit(0)
    with pytest.raises(RuntimeError, match="timed out"):
        gemm.check()
    gemm.clear()
    z1, _ = conv.forward(gemm, x)
    torch.cuda.synchronize()
    gemm.check()
    assert torch.equal(z0, z1)


@pytest.mark.parametrize("B,H,W,cout", [(1, 1, 2, 64), (2, 2, 4, 40), (3, 5, 6, 64), (1, 33, 258, 56),
                                        (2, 130, 64, 64), (1, 16, 31, 64), (5, 40, 20, 64)])
def test_pixel_pairs_of_32_channels_match_im2col(cuda_lib, B, H, W, cout):
    """Stride 2 from 32 channels: rows of pixel pairs (an odd width takes the taps one by
    one), bit for bit, and a wait that runs out is reported."""
    import torch
    from diffsplat_b200 import nn
    gen = torch.Generator().manual_seed(H * W)
    conv = nn.Conv3x3(32, cout, 2, gen=gen)
    conv.b.copy_(torch.randn(cout, generator=gen))
    x = torch.randn(B, H, W, 32, generator=gen).to(torch.bfloat16).cuda()
    gemm = nn.Gemm()
    nn.set_spin_limit(1)
    try:
        conv.forward(gemm, x)
        torch.cuda.synchronize()
    finally:
        nn.set_spin_limit(0)
    with pytest.raises(RuntimeError, match="timed out"):
        gemm.check()
    gemm.clear()
    z, y = conv.forward(gemm, x)
    col, _ = nn.im2col(x, 2, conv.kp)
    torch.cuda.synchronize()
    gemm.check()
    want_z, want_y = gemm(col, conv.w16, nn.EPI_BIAS_GELU, bias=conv.b)
    assert torch.equal(z.view(want_z.shape), want_z) and torch.equal(y.view(want_y.shape), want_y)
