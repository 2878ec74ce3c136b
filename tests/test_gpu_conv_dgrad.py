"""The input gradient of the implicit convolution is that of the GEMM dz . w with
col2im, bit for bit: each tap's products are one tensor-core sum, the taps are added in
FP32 in order, and a tap that reads past dz adds nothing (an infinite weight does not turn
the border into NaN)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,cin,cout", [
    (8, 1, 1, 64, 8), (8, 3, 2, 32, 56), (8, 17, 23, 32, 72), (8, 16, 16, 64, 128),
    (2, 31, 32, 128, 264), (1, 64, 200, 256, 256), (16, 8, 8, 320, 320), (8, 2, 9, 192, 2048)])
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("inf", [False, True])
def test_dgrad_equals_gemm_and_col2im(cuda_lib, B, H, W, cin, cout, stride, inf):
    import torch

    from diffsplat_b200 import nn
    gen = torch.Generator().manual_seed(cin + cout + H)
    conv = nn.Conv3x3(cin, cout, stride, gen=gen)
    if inf:  # corner taps: the border pixels read past dz through them
        conv.w16[0, 0] = float("inf")
        conv.w16[1, 8 * cin + 5] = -float("inf")
    x = torch.randn(B, H, W, cin, generator=gen).to(torch.bfloat16).cuda()
    zprev = torch.randn(B, H, W, cin, generator=gen).to(torch.bfloat16).cuda()
    gemm = nn.Gemm()
    z, _ = conv.forward(gemm, x)
    dz = torch.randn(z.shape, generator=gen).to(torch.bfloat16).cuda()
    assert dz.numel() // cout % 8 == 0
    dcol = gemm(dz.view(-1, cout), nn.transpose(conv.w16))
    for zp in (None, zprev):
        dx = conv.backward(gemm, dz, z_prev=zp)
        want = nn.col2im(dcol, x.shape, stride, zp)
        assert conv.col is None  # the implicit path ran
        assert torch.equal(dx.view(torch.int16), want.view(torch.int16))
    torch.cuda.synchronize()
    gemm.check()
