"""Covariance and position gradients of splats much thinner than a pixel, one by one,
against the FP64 recurrence on the GPU's own forward state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [2.0, 0.3, 0.1, 0.03, 0.01, 0.003])
@pytest.mark.parametrize("shape", ["round", "flat", "upright"])
def test_gradients_of_thin_splats(cuda_lib, sigma, shape):
    import torch

    from diffsplat_b200 import _lib as L, api
    from oracle import oracle as O
    # A power of two, so that pixel centres are exact in FP32; rows (and columns) of every
    # place in an 8x8 block; far enough apart to share no pixel
    N = 256
    step = 27 if sigma > 1 else 5
    at = np.arange(8, N - 8, step)
    r = np.random.default_rng(3)
    n = len(at)
    cx = at + r.uniform(-1.5, 1.5, n) * sigma if shape != "flat" else r.uniform(60, 190, n)
    cy = r.permutation(at) + r.uniform(-1.5, 1.5, n) * sigma if shape != "upright" else r.uniform(60, 190, n)
    sx = 5.0 if shape == "flat" else sigma
    sy = 5.0 if shape == "upright" else sigma
    S = np.zeros((10, n), np.float32)
    S[0] = (2 * cx + 1) / N - 1
    S[1] = 1 - (2 * cy + 1) / N
    S[2] = r.uniform(-0.9, 0.9, n)
    S[3], S[5] = (2 * sx / N) ** 2, (2 * sy / N) ** 2
    S[6:9] = r.uniform(0.2, 1, (3, n))
    S[9] = r.uniform(0.5, 0.9, n)
    S2 = torch.from_numpy(S).cuda()
    g = (0.5 + torch.rand(N, N, 3, generator=torch.Generator().manual_seed(5))).cuda()
    ras = api.Rasterizer(N, N, n, 1 << 18)
    ras.forward(S2)
    G2 = ras.backward(S2, g).cpu().numpy().astype(np.float64)
    torch.cuda.synchronize()
    ids, ranges = ras.download(L.DS_RASTER_IDS), ras.download(L.DS_RASTER_RANGES)
    want = O.composite_backward(S.astype(np.float64), N, N, ids, ranges.reshape(-1, 2),
                                ras.download(L.DS_RASTER_ALPHAS).reshape(N, N),
                                ras.download(L.DS_RASTER_LAST_IDS).reshape(N, N),
                                g.cpu().numpy().astype(np.float64))
    # Every term of a sum has the same sign (one splat a pixel, all weights positive), but
    # for the position's and cov xy's, held against what their terms add up to.  In units
    # u = 2^-24: the conic is within 4 u, an offset 1, dist2 9, so the exponent of at most
    # ln(255 x 0.9) = 5.4 is within 60 u and the exponential 64; a squared slope 12, colour
    # and transmittance (1 - alpha from 0.1 up) 25, products and sums 15: 116 u = 7e-6.
    tol = 1e-5
    seen = np.abs(want[9]) > 0
    if 6 * max(sx, sy) < 1:  # less than a pixel across in both directions: culled
        assert not G2.any() and not seen.any()
        return
    assert seen.sum() >= n // 2
    for row in (3, 5, 9):
        assert (np.abs(G2[row] - want[row])[seen] <= tol * np.abs(want[row])[seen]).all(), row
    # Cauchy-Schwarz over the terms: |sum s u| <= sqrt(sum s * sum s u^2)
    s = np.abs(want[9]) * S[9]
    for row, bound in ((0, np.sqrt(2 * s * np.abs(want[3]))), (1, np.sqrt(2 * s * np.abs(want[5]))),
                       (4, 2 * np.sqrt(np.abs(want[3] * want[5])))):
        assert (np.abs(G2[row] - want[row])[seen] <= tol * bound[seen]).all(), row
