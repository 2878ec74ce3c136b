"""A resize that runs out of memory at any of its allocations leaves no half of a grid:
calls that need one are refused until a resize succeeds, and that one gives the lists and
image of a fresh object.  The size asked for has more tiles along x than the bins hold, so the
buffers of sorted pairs are allocated with it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 16400, 16  # 1025 tiles


def _until_it_succeeds(resize, refused):
    from diffsplat_b200 import _lib as L
    k = 0
    try:
        while True:
            assert k < 100
            L.lib().ds_debug_fail_allocations_after(k)
            st = resize()
            L.lib().ds_debug_fail_allocations_after(-1)
            if st == L.DS_OK:
                return k
            assert st == L.DS_ERR_OOM
            refused()
            k += 1
    finally:
        L.lib().ds_debug_fail_allocations_after(-1)


def test_raster_resize_out_of_memory(cuda_lib):
    import torch

    from diffsplat_b200 import _lib as L, api
    n = 400
    r = np.random.default_rng(2)
    S = np.zeros((10, n), np.float32)
    S[0:3] = r.uniform(-0.9, 0.9, (3, n))
    S[3] = S[5] = r.uniform(1e-3, 4e-2, n) ** 2
    S[6:10] = 0.5
    S2 = torch.from_numpy(S).cuda()
    fresh = api.Rasterizer(W, H, n, 1 << 18)
    want = fresh.forward(S2).cpu()
    ras = api.Rasterizer(96, 64, n, 1 << 18)
    ras.forward(S2)
    out = torch.empty(H, W, 3, device="cuda")
    view = api.s2_view(S2)

    def refused():
        assert L.lib().ds_raster_forward(ras.h, C.byref(view), out.data_ptr(), None) == L.DS_ERR_STATE
        assert L.lib().ds_raster_backward(ras.h, C.byref(view), out.data_ptr(), C.byref(view),
                                          None) == L.DS_ERR_STATE

    assert _until_it_succeeds(lambda: L.lib().ds_raster_resize(ras.h, W, H), refused) > 6
    assert L.lib().ds_raster_forward(ras.h, C.byref(view), out.data_ptr(), None) == L.DS_OK
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want)
    assert L.lib().ds_raster_resize(ras.h, 16 * 65535 + 1, 16) == L.DS_ERR_ARG  # keeps its grid
    assert L.lib().ds_raster_forward(ras.h, C.byref(view), out.data_ptr(), None) == L.DS_OK
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want)


def test_renderer_resize_out_of_memory(cuda_lib):
    import torch

    from diffsplat_b200 import _lib as L, api
    from diffsplat_b200.scenes import small_problem
    big = small_problem(W, H, 300, seed=57)
    P = torch.tensor(big.params, device="cuda")
    fresh = api.Renderer(W, H, 300, 0, max_isects=1 << 18)
    fresh.set_params(P)
    want = fresh.render(big.pv, big.cam).cpu()
    r = api.Renderer(96, 64, 300, 0, max_isects=1 << 18)
    r.set_params(P)

    def refused():
        assert L.lib().ds_renderer_render(r.h, L.fptr(big.pv), L.fptr(big.cam), None) == L.DS_ERR_STATE

    assert _until_it_succeeds(lambda: L.lib().ds_renderer_resize(r.h, W, H), refused) > 6
    r.width, r.height = W, H
    img = r.render(big.pv, big.cam).cpu()
    assert torch.equal(img, want)
