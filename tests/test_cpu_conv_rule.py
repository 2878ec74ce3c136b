"""Conv3x3 hands the implicit kernels, which get bare pointers, only what fits the layer:
everything else goes through im2col and the GEMM, whose shape checks refuse what they
always refused (a gradient of too few pixels would be read past its end)."""
import pytest
import torch

from diffsplat_b200 import nn

BF16 = torch.bfloat16


def _conv(cin, cout, stride=1):
    c = nn.Conv3x3.__new__(nn.Conv3x3)  # no device
    c.cin, c.cout, c.stride, c.kp = cin, cout, stride, nn.kpad(cin)
    c.w16 = torch.zeros(cout, c.kp, dtype=BF16)
    c.b, c.gw = torch.zeros(cout), torch.zeros(cout, c.kp)
    c.col = None
    return c


def _x(*shape, dtype=BF16):
    return torch.zeros(shape, dtype=dtype)


@pytest.mark.parametrize("x,ok", [
    (_x(2, 8, 8, 64), True), (_x(2, 8, 8, 32), False), (_x(2, 8, 8, 128), False),
    (_x(2, 8, 8, 64, dtype=torch.float32), False), (_x(2, 8, 8, 64, dtype=torch.float16), False),
    (_x(2, 64, 8, 8).permute(0, 2, 3, 1), False), (_x(2, 8, 8, 128)[..., ::2], False)])
def test_forward_takes_only_inputs_of_the_layer(x, ok):
    assert _conv(64, 64)._implicit(x, rgb=True) == ok


@pytest.mark.parametrize("stride,pixels", [(1, 2 * 9 * 7), (2, 2 * 5 * 4)])
def test_backward_takes_only_gradients_of_all_pixels(stride, pixels):
    c = _conv(64, 56, stride)
    c.x, c.in_shape = _x(2, 9, 7, 64), (2, 9, 7, 64)
    z = _x(2, 9, 7, 64)
    for rows, ok in ((pixels, True), (pixels - 8, False), (pixels + 8, False), (8, False)):
        assert c._implicit_backward(_x(rows, 56), None) == ok
        assert c._implicit_backward(_x(rows, 56), z) == ok
    assert not c._implicit_backward(_x(pixels, 56, dtype=torch.float32), z)
    assert not c._implicit_backward(_x(pixels, 56), z.float())
    c.col = _x(pixels, c.kp)  # the forward went through im2col
    assert not c._implicit_backward(_x(pixels, 56), z)
