"""Backward of the three-channel layer on both sides of the size up to which the forward keeps
the im2col matrix: weight and bias gradients of the input as the forward saw it, those of
transposes and GEMM bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(8, 5, 7), (8, 64, 127), (8, 64, 128)])
@pytest.mark.parametrize("keep", [False, True])
def test_gradients_of_the_input_as_it_was(cuda_lib, B, H, W, keep):
    import torch

    from diffsplat_b200 import nn
    gen = torch.Generator().manual_seed(H)
    conv = nn.Conv3x3(3, 32, 1, gen=gen)
    gemm = nn.Gemm()
    x = torch.randn(B, H, W, 3, generator=gen).to(torch.bfloat16).cuda()
    col, _ = nn.im2col(x, 1, conv.kp)
    z, _ = conv.forward(gemm, x, keep=keep)
    assert conv.col is None
    if not keep:
        x.fill_(float("nan"))
    dz = torch.randn(z.shape, generator=gen).to(torch.bfloat16).cuda()
    assert conv.backward(gemm, dz, need_dx=False) is None
    M = B * H * W
    want = gemm(nn.transpose(dz.view(M, 32)), nn.transpose(col), splits=max(1, min(64, M // 4096)))
    torch.cuda.synchronize()
    gemm.check()
    assert torch.equal(conv.gw, want)
    assert torch.allclose(conv.gb, dz.float().sum((0, 1, 2)), rtol=1e-4, atol=1e-2)
