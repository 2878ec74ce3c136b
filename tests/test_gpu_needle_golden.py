"""Splat2D gradients of long thin splats at all angles equal the recorded ones of the
per-pixel formula in FP32, d dist2 / d(cov xy) = -2 (b dist2 + dx dy / det): its rounding
(1e-4 of the norm here, up to most of a single scale gradient further on) is part of the
result, which u w, equal in exact arithmetic, does not reproduce.

tests/golden/needles_grad2d.npz holds the [10, 240] gradients of scene() from the butterfly
form of the composite backward (one pixel per lane, nine sums a hit).  Sums in another order
differ by some 1e-7; the bound is the 2e-5 of the norm that FP32 results of one scene are
held to, and 8e-4 for the worst single value."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden" / "needles_grad2d.npz"
W, H = 200, 152


def scene():
    r, n = np.random.default_rng(77), 240
    S = np.zeros((10, n), np.float32)
    S[0:2] = r.uniform(-.95, .95, (2, n))
    S[2] = r.permutation(n) / n - .5
    long = np.exp(r.uniform(np.log(.02), np.log(.3), n))
    short = long / np.exp(r.uniform(np.log(4), np.log(90), n))
    th = r.uniform(0, np.pi, n)
    c, s = np.cos(th), np.sin(th)
    S[3] = (c * long) ** 2 + (s * short) ** 2
    S[4] = c * s * (long ** 2 - short ** 2)
    S[5] = (s * long) ** 2 + (c * short) ** 2
    S[6:9] = r.uniform(0, 1, (3, n))
    S[9] = r.uniform(.05, .9, n)
    return S, r.standard_normal((H, W, 3)).astype(np.float32)


def test_gradients_of_needles(cuda_lib):
    import torch

    from diffsplat_b200 import api
    S, g = scene()
    ras = api.Rasterizer(W, H, S.shape[1], 1 << 18)
    S2 = torch.from_numpy(S).cuda()
    ras.forward(S2)
    G = ras.backward(S2, torch.from_numpy(g).cuda())
    torch.cuda.synchronize()
    G, want = G.cpu().numpy().astype(np.float64), np.load(GOLDEN)["G"].astype(np.float64)
    for row in (0, 1, 3, 4, 5, 6, 7, 8, 9):
        d, rms = np.abs(G[row] - want[row]), np.sqrt((want[row] ** 2).mean())
        assert np.linalg.norm(d) <= 2e-5 * np.linalg.norm(want[row]), row
        assert (d / np.maximum(rms, np.abs(want[row]))).max() <= 8e-4, row
