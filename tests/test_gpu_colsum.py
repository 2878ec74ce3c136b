"""Column sums add the rows of a chunk one after another and then the chunks, in FP32: the
same values bit for bit at every width, alignment and remainder."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,C", [(1, 8), (7, 56), (1000, 3), (255, 264), (5000, 200), (777, 8),
                                 (70_001, 520), (151_553, 32), (131_072, 64)])
@pytest.mark.parametrize("offset", [0, 1])
def test_sums_in_row_order(cuda_lib, M, C, offset):
    import torch

    from diffsplat_b200 import nn
    flat = torch.randn(M * C + offset, generator=torch.Generator().manual_seed(M + C))
    a = flat.to(torch.bfloat16).cuda()[offset:].view(M, C)
    got = nn.colsum(a)
    rows = a.float().cpu().numpy()
    chunk = max(256, -(-M // (148 * 4)))
    parts = -(-M // chunk)
    padded = np.zeros((parts * chunk, C), np.float32)
    padded[:M] = rows
    part = np.zeros((parts, C), np.float32)
    for r in range(chunk):
        part += padded[r::chunk]
    want = np.zeros(C, np.float32)
    for k in range(parts):
        want += part[k]
    assert np.array_equal(got.cpu().numpy(), want)
