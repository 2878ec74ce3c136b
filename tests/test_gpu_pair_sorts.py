"""The sorts of (tile, splat) pairs, which rasterizers for more than 65536 splats use
(counting up to 8192 tiles, radix passes above), reached by such a capacity with scenes small
enough to list by bins too: both must give the same lists, image and gradients, ordered by
tile, depth and id.  Scenes up to 65536 splats no longer reach them by themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOST_BY_BINS = 65536


def _run(W, H, S2, capacity, cap):
    import torch

    from diffsplat_b200 import _lib as L, api
    ras = api.Rasterizer(W, H, capacity, cap)
    img = ras.forward(S2).clone()
    G2 = ras.backward(S2, torch.ones(H, W, 3, device="cuda") * 0.5 + img).cpu().numpy()
    torch.cuda.synchronize()
    out = dict(keys=ras.download(L.DS_RASTER_KEYS), ids=ras.download(L.DS_RASTER_IDS),
               ranges=ras.download(L.DS_RASTER_RANGES), image=img.cpu().numpy(), G2=G2,
               pairs=ras.isect_count())
    ras.close()
    return out


def _splats(n, seed, log_scale):
    import torch
    r = np.random.default_rng(seed)
    S = np.zeros((10, n), np.float32)
    S[0:2] = r.uniform(-1.1, 1.1, (2, n))
    S[2] = -0.5 + r.integers(0, max(2, n // 3), n) / n  # equal depths among them
    S[3], S[5] = np.exp(2 * (log_scale + 0.5 * r.standard_normal((2, n))))
    S[6:9] = r.uniform(0, 1, (3, n))
    S[9] = r.uniform(0.02, 0.9, n)
    return torch.from_numpy(S).cuda()


#        W,   H,      n, log-scale, capacity of pairs, at least so many pairs
CASES = [(160, 90, 600, -2.0, 1 << 20, 1),
         (1920, 1080, 6000, -3.0, 1 << 23, 1),
         (2048, 1024, 6000, -3.0, 1 << 23, 1),               # 8192 tiles: the last counted
         (2064, 1024, 6000, -3.0, 1 << 23, 1),               # 8256: radix passes
         (1024, 1024, 20000, -1.2, 1 << 25, 296 * 65535),    # chunks past 16-bit offsets
         (1920, 1080, 65536, -2.2, 1 << 26, 296 * 65535),
         (512, 512, 8000, -2.0, 100_000, 100_000)]           # more pairs than fit


@pytest.mark.parametrize("W,H,n,scale,cap,least", CASES)
def test_sorted_pairs_equal_lists_by_bins(cuda_lib, W, H, n, scale, cap, least):
    S2 = _splats(n, n, scale)
    me = _run(W, H, S2, MOST_BY_BINS + 1, cap)
    want = _run(W, H, S2, n, cap)
    assert me["pairs"] == want["pairs"] >= least and (me["pairs"] > cap) == (cap == 100_000)
    for k in ("keys", "ids", "ranges"):
        assert np.array_equal(me[k], want[k]), k
    for k in ("image", "G2"):
        assert np.array_equal(me[k].view(np.uint32), want[k].view(np.uint32)), k
    kept = min(me["pairs"], cap)
    k, i = me["keys"][:kept].astype(np.int64), me["ids"][:kept].astype(np.int64)
    assert np.all((k[1:] > k[:-1]) | ((k[1:] == k[:-1]) & (i[1:] > i[:-1])))
