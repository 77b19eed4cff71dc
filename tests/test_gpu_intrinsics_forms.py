"""refine_intrinsics in its two forms: cameras that go through their loops in
step, each alone in its problem, and the same cameras as one block each, among
many small ones. A camera's result does not depend on the others, and both
forms add in one order, so the results are the same bits; the small cameras are
held against the oracle (1e-6 relative, as in test_gpu_intrinsics.py)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native
from sfmtory_gb300.problem import Problem, project

pytestmark = pytest.mark.gpu

TRUE = {abi.PINHOLE: [1200.0, 1190.0, 800.0, 600.0, 0, 0, 0, 0],
        abi.SIMPLE_RADIAL: [1200.0, 800.0, 600.0, 0.03, 0, 0, 0, 0],
        abi.OPENCV: [1200.0, 1190.0, 800.0, 600.0, 0.05, -0.02, 1e-3, -1e-3]}


def _cameras(counts, models, seed):
    rng = np.random.default_rng(seed)
    n, nC = sum(counts), len(counts)
    X = np.stack([rng.uniform(-2, 2, n), rng.uniform(-2, 2, n), rng.uniform(4, 8, n)], 1)
    X[rng.choice(n, n // 50, replace=False), 2] *= -1.0  # behind their camera
    cam = np.repeat(np.arange(nC, dtype=np.int32), counts)
    model = np.array(models, np.int32)
    true = np.array([TRUE[m] for m in models], np.float64)
    front = X.copy()
    front[:, 2] = np.abs(front[:, 2])
    xy = project(model[cam], true[cam], front) + rng.normal(0.0, 0.5, (n, 2))
    true[:, 0] *= 1.02
    o = rng.permutation(n)
    return Problem(camera_of_image=np.arange(nC, dtype=np.int32), camera_model=model, camera_params=true,
                   poses=np.tile([1.0, 0, 0, 0, 0, 0, 0], (nC, 1)), points=X, obs_image=cam[o],
                   obs_point=o.astype(np.int32), obs_xy=xy[o])


def _alone(p, c):
    keep = p.obs_image == c
    return p.copy(camera_of_image=np.zeros(1, np.int32), camera_model=p.camera_model[c:c + 1],
                  camera_params=p.camera_params[c:c + 1], poses=p.poses[c:c + 1],
                  obs_image=np.zeros(keep.sum(), np.int32), obs_point=p.obs_point[keep], obs_xy=p.obs_xy[keep])


@pytest.mark.parametrize("loss", [abi.LOSS_NONE, abi.LOSS_HUBER])
def test_the_two_forms_give_the_same_bits(oracle_lib, loss):
    kinds = list(TRUE)
    large = [129, 255, 256, 257, 700, 1000]
    counts = large + [8, 7, 60, 127, 128] * 80
    p = _cameras(counts, [kinds[k % 3] for k in range(len(counts))], seed=int(loss))
    kw = dict(robust_loss=loss, loss_scale_px=2.0, max_iterations=20)
    g = native.refine_intrinsics_arrays(p, **kw)
    for c in range(len(large)):
        assert np.array_equal(g[c], native.refine_intrinsics_arrays(_alone(p, c), **kw)[0]), c
    kw["max_iterations"] = 4
    g, r = native.refine_intrinsics_arrays(p, **kw), oracle_lib.refine_intrinsics(p, **kw)
    for c, n in enumerate(counts):
        if n < 8:
            assert np.array_equal(g[c], p.camera_params[c])
        elif p.camera_model[c] == abi.PINHOLE:  # linear in the parameters: no noise of the differences
            assert (np.abs(g[c] - r[c]) / np.maximum(np.abs(r[c]), 1.0)).max() <= 1e-6, (c, g[c], r[c])
