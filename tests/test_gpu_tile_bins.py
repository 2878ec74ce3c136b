"""Tile lists by bins of 8 x 8 tiles (and, for many splats over many bins, by the
counting sort of the pairs) against the radix passes: partial bins, chunks with a
remainder, splats over everything, none at all, and pairs beyond the capacity."""
import numpy as np
import pytest

from tests.test_gpu_tile_sort import _lists, _radix_lists

pytestmark = pytest.mark.gpu

#        W,   H,      n, log-scale, capacity
CASES = [(8, 8, 1, -2.5, 1 << 16),
         (16, 16, 33, -1.0, 1 << 16),
         (130, 70, 65, -0.5, 1 << 16),        # one bin and a little
         (1030, 40, 700, -2.0, 1 << 20),      # a row of bins, the last one tile wide
         (40, 1500, 4097, -3.0, 1 << 20),
         (512, 512, 20001, -3.5, 1 << 22),    # sparse: few splats per tile and group
         (800, 600, 3000, -1.0, 1 << 23),     # dense
         (800, 600, 3000, -1.0, 12345),       # more pairs than fit
         (1920, 1080, 260_000, -5.0, 1 << 22)]  # past the bins: the counting sort


@pytest.mark.parametrize("W,H,n,scale,cap", CASES)
def test_lists_equal_the_radix_paths(cuda_lib, tmp_path, W, H, n, scale, cap):
    _, me = _lists(W, H, n, 3, scale, cap)
    rx = _radix_lists(tmp_path, W, H, n, 3, scale, cap)
    for k in ("keys", "ids", "ranges"):
        assert np.array_equal(me[k], rx[k]), k
    assert np.array_equal(me["image"].view(np.uint32), rx["image"].view(np.uint32))
    assert np.array_equal(me["G2"].view(np.uint32), rx["G2"].view(np.uint32))


def test_batch_lists_do_not_depend_on_the_company(cuda_lib):
    """An instance's image and parameters after two steps are those of a batch of
    its own: 300 instances take two digits of the instance sort."""
    import torch

    from diffsplat_b200 import api
    from diffsplat_b200.scenes import small_problem
    sizes = [(40 + 8 * (k % 7), 24 + 8 * (k % 5), 50 + 13 * (k % 11)) for k in range(300)]
    probs = [small_problem(w, h, n, seed=k % 17) for k, (w, h, n) in enumerate(sizes)]

    def fit(which):
        b = api.Batch([sizes[k] for k in which], storage=0, max_isects=1 << 22)
        for j, k in enumerate(which):
            b.set_params(j, probs[k].params)
            b.set_target(j, torch.from_numpy(probs[k].target).cuda())
            b.set_camera(j, probs[k].pv, probs[k].cam)
        b.step(2)
        torch.cuda.synchronize()
        assert b.status()[0] == 0
        return [(b.image(j).cpu().numpy(), b.instance_params(j).cpu().numpy())
                for j in range(len(which))]

    many = fit(range(300))
    for k in (0, 131, 299):
        img, par = fit([k])[0]
        assert np.array_equal(img, many[k][0]) and np.array_equal(par, many[k][1])


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 2049, 4096, 8192, 8193, 20000, 65535, 65536, 65537])
@pytest.mark.parametrize("depths", [1, 7, 100_000])
def test_order_is_by_depth_then_id(cuda_lib, n, depths):
    """The sorts of up to 8192 splats (by counting), of up to 65536 (one cluster) and of
    more: equal depths by id, depths that share all digits or few, splats in no tile
    among them."""
    import torch

    from diffsplat_b200 import _lib as L, api
    r = np.random.default_rng(n + depths)
    S = np.zeros((10, n), np.float32)
    S[0:2] = r.uniform(-1.2, 1.2, (2, n))  # some centres outside: culled
    S[2] = -0.5 + r.integers(0, depths, n) / depths
    S[3] = S[5] = r.uniform(1e-3, 4e-2, n) ** 2
    S[6:10] = 0.5
    S2 = torch.from_numpy(S).cuda()
    ras = api.Rasterizer(200, 120, n, 1 << 22)
    ras.forward(S2)
    keys, ids = ras.download(L.DS_RASTER_KEYS), ras.download(L.DS_RASTER_IDS)
    counts = ras.download(L.DS_RASTER_COUNTS, n)
    assert len(keys) == counts.sum() and ras.status()[0] == 0
    k, i = keys.astype(np.int64), ids.astype(np.int64)
    assert np.all((k[1:] > k[:-1]) | ((k[1:] == k[:-1]) & (i[1:] > i[:-1])))
    assert np.array_equal(np.bincount(i, minlength=n), counts)
    ranges = ras.download(L.DS_RASTER_RANGES).reshape(-1, 2)
    assert np.array_equal(np.bincount(k >> 32, minlength=len(ranges)), ranges[:, 1] - ranges[:, 0])
