"""A gradient that does not fit the layer's output is refused, as by im2col + GEMM."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,dtype,need_dx", [(56, "bfloat16", True), (72, "bfloat16", False),
                                                (64, "float32", True)])
def test_gradient_that_does_not_fit_is_refused(cuda_lib, rows, dtype, need_dx):
    import torch

    from diffsplat_b200 import nn
    gemm = nn.Gemm()
    conv = nn.Conv3x3(64, 64, gen=torch.Generator().manual_seed(0))
    x = torch.randn(1, 8, 8, 64).to(torch.bfloat16).cuda()
    conv.forward(gemm, x)
    dz = torch.zeros(rows, 64, dtype=getattr(torch, dtype), device="cuda")
    with pytest.raises(AssertionError):
        conv.backward(gemm, dz, need_dx=need_dx)
    torch.cuda.synchronize()
    gemm.check()
