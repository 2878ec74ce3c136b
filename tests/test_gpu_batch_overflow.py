"""A batch with more pairs than max_isects drops the deepest pairs of all instances,
whichever way its tile lists are built: images, losses and parameters are those of the
radix passes, whose order is by depth alone."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def run(count, cap):
    import torch

    from diffsplat_b200 import api
    from diffsplat_b200.scenes import small_problem
    sizes = [(40 + 8 * (k % 7), 24 + 8 * (k % 5), 50 + 13 * (k % 11)) for k in range(count)]
    probs = [small_problem(w, h, n, seed=k % 17) for k, (w, h, n) in enumerate(sizes)]
    b = api.Batch(sizes, storage=0, max_isects=cap)
    for k, p in enumerate(probs):
        b.set_params(k, p.params)
        b.set_target(k, torch.from_numpy(p.target).cuda())
        b.set_camera(k, p.pv, p.cam)
    b.step(2)
    torch.cuda.synchronize()
    pairs = b.counters()["n_isects"]
    return dict(pairs=pairs, status=b.status()[0], losses=np.asarray(b.losses()),
                images=np.concatenate([b.image(k).cpu().numpy().ravel() for k in range(count)]),
                params=b.params.cpu().numpy())


@pytest.mark.parametrize("count,cap", [(1, 40), (1, 1 << 16), (5, 199), (5, 1),
                                       (300, 30_001), (300, 1 << 20)])
def test_overflow_drops_the_deepest_pairs(cuda_lib, tmp_path, count, cap):
    dst = tmp_path / "radix.npz"
    code = ("import sys; sys.path.insert(0, %r)\nimport numpy as np\n"
            "from tests.test_gpu_batch_overflow import run\n"
            "np.savez(%r, **run(%d, %d))\n" % (str(ROOT), str(dst), count, cap))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, DS_TILE_SORT="radix"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    want, me = np.load(dst), run(count, cap)
    over = me["pairs"] > cap
    assert over == (cap < 1 << 16) and (me["status"] != 0) == over
    for k in ("pairs", "status", "losses", "images", "params"):
        assert np.array_equal(me[k], want[k]), k
