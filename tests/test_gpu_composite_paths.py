"""The composite backward's two pixel loops (plain splats, and those that may reach
alpha 0.99, whose conic is nearly singular or whose pixels ended opaque) against the
FP64 recurrence on the GPU's own forward state."""
import numpy as np
import pytest

from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def _splats(kind, n, W, H, seed):
    """Splat2D rows [10, n]: sigma from a third of a pixel to a third of the image."""
    r = np.random.default_rng(seed)
    S = np.zeros((10, n))
    S[0:2] = r.uniform(-1, 1, (2, n))
    S[2] = r.uniform(-0.9, 0.9, n)
    long = np.exp(r.uniform(np.log(0.7 / W), np.log(0.6), n))
    aspect = r.uniform(1, 8, n)
    needle = np.zeros(n, bool)
    if kind == "needle":
        needle = r.random(n) < 0.5
        long[needle] = r.uniform(0.2, 0.4, needle.sum())
        aspect[needle] = r.uniform(105, 115, needle.sum())
    th = r.uniform(0, np.pi, n)
    short = long / aspect
    c, s = np.cos(th), np.sin(th)
    S[3] = (c * long) ** 2 + (s * short) ** 2
    S[4] = c * s * (long ** 2 - short ** 2)
    S[5] = (s * long) ** 2 + (c * short) ** 2
    S[6:9] = r.uniform(0, 1, (3, n))
    S[9] = r.uniform(0.02, 0.9, n)
    if kind in ("opaque", "needle"):
        high = r.random(n) < 0.4
        S[9, high] = r.uniform(0.99, 0.9999, high.sum())
    return S.astype(np.float32)


@pytest.mark.parametrize("kind,W,H,n", [("plain", 16, 16, 5), ("plain", 40, 23, 300),
                                        ("opaque", 40, 23, 300), ("opaque", 129, 65, 900),
                                        ("needle", 64, 64, 200)])
def test_backward_against_fp64_recurrence(cuda_lib, kind, W, H, n):
    import torch

    from diffsplat_b200 import _lib as L, api
    from oracle import oracle as O
    S2 = torch.from_numpy(_splats(kind, n, W, H, 11)).cuda()
    g = torch.randn(H, W, 3, generator=torch.Generator().manual_seed(5)).cuda()
    r = api.Rasterizer(W, H, n, 1 << 18)
    img = r.forward(S2)
    G2 = r.backward(S2, g).cpu().numpy()
    torch.cuda.synchronize()
    ids, ranges = r.download(L.DS_RASTER_IDS), r.download(L.DS_RASTER_RANGES)
    want = O.composite_backward(S2.cpu().numpy().astype(np.float64), W, H, ids,
                                ranges.reshape(-1, 2), r.download(L.DS_RASTER_ALPHAS).reshape(H, W),
                                r.download(L.DS_RASTER_LAST_IDS).reshape(H, W),
                                g.cpu().numpy().astype(np.float64))
    assert torch.isfinite(img).all()
    # 2e-4 as for the rasterizer's other comparisons with this recurrence; a needle of
    # aspect 115 cancels all but 1 / 115^2 of its quadratic form, in four operations, and
    # the exponent reaches 5: 115^2 2^-24 4 5 = 1.6e-2
    tol = 2e-2 if kind == "needle" else 2e-4
    for row in (0, 1, 3, 4, 5, 6, 7, 8, 9):
        assert rel_err(G2[row], want[row]) <= tol, f"row {row}"
