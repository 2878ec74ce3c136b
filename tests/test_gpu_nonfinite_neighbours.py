"""A splat whose colour is infinite or NaN spoils the gradients of the splats that share a
pixel with it and of no others, also not of those in the same 8x8 block of pixels."""
import numpy as np
import pytest

from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def _grads(S, mode):
    import torch

    from diffsplat_b200 import api
    ras = api.Rasterizer(32, 32, S.shape[1], 1 << 14)
    ras.set_grad_mode(mode)
    S2 = torch.from_numpy(S).cuda()
    img = ras.forward(S2).clone()
    g = torch.randn(32, 32, 3, generator=torch.Generator().manual_seed(3)).cuda()
    G = ras.backward(S2, g)
    torch.cuda.synchronize()
    return img.cpu().numpy(), G.cpu().numpy()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38])
@pytest.mark.parametrize("mode", [0, 1])
def test_only_splats_that_share_a_pixel(cuda_lib, value, mode):
    # splats of sigma 0.4 pixels: one covers at most the 3x3 pixels around it
    at = [(c, r) for r in range(1, 32, 4) for c in range(1, 32, 4)]
    n = len(at)
    rng = np.random.default_rng(1)
    S = np.zeros((10, n), np.float32)
    S[0] = [(2 * c + 1) / 32 - 1 for c, _ in at]
    S[1] = [1 - (2 * r + 1) / 32 for _, r in at]
    S[2] = rng.permutation(n) / n - 0.5  # some spoilt ones behind their neighbours, some before
    S[3] = S[5] = (0.4 / 16) ** 2
    S[6:9] = rng.uniform(0, 1, (3, n))
    S[9] = 0.8
    img0, G0 = _grads(S, mode)
    assert np.isfinite(G0).all() and (G0[9] != 0).all()
    spoilt = rng.choice(n, n // 8, replace=False)
    S[rng.integers(6, 9, len(spoilt)), spoilt] = value
    img, G = _grads(S, mode)
    clean = np.setdiff1d(np.arange(n), spoilt)
    assert np.isfinite(G[:, clean]).all()
    # the pixel loop with selects multiplies in another order: a few 2^-24 of each term, of which
    # up to nine of either sign make a sum
    for row in (0, 1, 3, 4, 5, 6, 7, 8, 9):
        assert rel_err(G[row, clean], G0[row, clean]) <= 1e-5, row
    if not abs(value) < 3.4e38:
        assert not np.isfinite(G[9, spoilt]).any()
