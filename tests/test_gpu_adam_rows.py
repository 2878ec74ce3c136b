"""Adam inside the fused step, where its rows are read four at a time and where they
cannot be (a splat count that is no multiple of 4), with and without SH rest rows."""
import numpy as np
import pytest

from diffsplat_b200.scenes import small_problem

pytestmark = pytest.mark.gpu

LRS = (1e-2, 2e-3, 3e-3, 4e-3, 5e-3, 6e-3)


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("degree", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 255, 256, 260, 1001])
def test_first_step_is_adam_of_the_steps_gradient(cuda_lib, n, degree, storage):
    from diffsplat_b200 import api
    import torch
    p = small_problem(96, 64, n, seed=4, sh_degree=degree)
    f = api.Fitter(96, 64, n, degree, lrs=LRS, keep_grads=True, storage=storage, eps=1e-6)
    f.set_params(p.params)
    f.set_target(torch.from_numpy(p.target).cuda())
    f.set_camera(p.pv, p.cam)
    before = f.params.cpu().numpy().astype(np.float64)
    f.step()
    torch.cuda.synchronize()
    after, g = f.params.cpu().numpy().astype(np.float64), f.grads().cpu().numpy().astype(np.float64)
    assert np.abs(g).max() > 0
    rows = np.arange(before.shape[0])
    lr = np.select([rows < 3, rows < 6, rows < 10, rows < 13, rows == 13],
                   [LRS[0], LRS[1], LRS[2], LRS[3], LRS[5]], LRS[4])[:, None]
    want = before - lr * g / (np.abs(g) + 1e-6)
    # one rounding of the parameter (2^-24) and FP32 arithmetic with the hardware's
    # square root and division (a few 2^-22) on an update of at most lr
    assert np.all(np.abs(after - want) <= 2.0 ** -23 * np.abs(want) + 2e-6 * lr)
    if storage == 0:
        m, v = (t.cpu().numpy() for t in f.moments())
        one = np.float32(1)  # the betas are FP32, 1 - 0.999 with them
        assert np.allclose(m, (one - np.float32(0.9)) * g, rtol=1e-6, atol=1e-30)
        assert np.allclose(v, (one - np.float32(0.999)) * g * g, rtol=1e-5, atol=1e-30)
