"""The composite backward takes its lists 64 or 256 splats at a time, by the number of
tiles and the capacity: the same gradients, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(160, 90, 300), (300, 300, 2000), (400, 800, 9000)])
def test_batch_lengths_agree(cuda_lib, shape):
    """Lists taken 64 and 256 splats at a time (grids of up to 296 tiles, or up to 4096 with a
    capacity of more than 65536 splats) give the same gradients, bit for bit."""
    import torch

    from diffsplat_b200 import api
    w, h, n = shape
    r = np.random.default_rng(n)
    S = np.zeros((10, n), np.float32)
    S[0:2] = r.uniform(-1, 1, (2, n))
    S[2] = r.uniform(-.9, .9, n)
    S[3], S[5] = np.exp(2 * r.normal(-3, .7, (2, n)))
    S[6:9] = r.uniform(0, 1, (3, n))
    S[9] = r.uniform(.05, 1, n)  # some past 0.99
    S2 = torch.from_numpy(S).cuda()
    g = torch.randn(h, w, 3, generator=torch.Generator().manual_seed(1)).cuda()
    out = []
    for capacity in (n, 70_000):
        ras = api.Rasterizer(w, h, capacity, 1 << 22)
        img = ras.forward(S2).clone()
        out.append((img, ras.backward(S2, g).clone()))
        torch.cuda.synchronize()
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])
