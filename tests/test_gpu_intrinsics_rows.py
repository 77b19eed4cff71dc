"""refine_intrinsics where its observation rows end: cameras with fewer
observations than it refines (7), the fewest (8), one short of, exactly and
one past a 128-observation row, and one whose rows pass the 2048 whose terms
are held at once, each against the oracle's restatement.

Bars: those of test_gpu_intrinsics.py (focal lengths and principal points
1e-6 relative); PINHOLE cameras, whose residual is linear in the parameters,
so the difference columns carry only the rounding of the pixel coordinates
(1e-13 px over a 2e-6 step: 1e-7 of a column of size 1, averaged over the
observations)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native
from sfmtory_gb300.problem import Problem, project

pytestmark = pytest.mark.gpu


def _scene(counts, seed):
    rng = np.random.default_rng(seed)
    n = sum(counts)
    X = np.stack([rng.uniform(-2, 2, n), rng.uniform(-2, 2, n), rng.uniform(4, 8, n)], 1)
    cam = np.repeat(np.arange(len(counts), dtype=np.int32), counts)
    true = np.zeros((len(counts), 8))
    true[:, :4] = [1200.0, 1190.0, 800.0, 600.0]
    xy = project(np.full(n, abi.PINHOLE), true[cam], X) + rng.normal(0.0, 0.5, (n, 2))
    start = true.copy()
    start[:, :2] *= 1.02
    poses = np.tile([1.0, 0, 0, 0, 0, 0, 0], (len(counts), 1))
    o = rng.permutation(n)
    return Problem(camera_of_image=np.arange(len(counts), dtype=np.int32),
                   camera_model=np.full(len(counts), abi.PINHOLE, np.int32), camera_params=start, poses=poses,
                   points=X, obs_image=cam[o], obs_point=o.astype(np.int32), obs_xy=xy[o])


@pytest.mark.parametrize("counts", [(8,), (7, 8, 127, 128, 129, 1, 1000), (300, 262144 + 130, 50, 262144 + 1)],
                         ids=["smallest", "row_ends", "past_the_held_rows"])
@pytest.mark.parametrize("loss", [abi.LOSS_NONE, abi.LOSS_HUBER])
def test_row_ends_match_oracle(oracle_lib, counts, loss):
    p = _scene(counts, seed=len(counts))
    kw = dict(robust_loss=loss, loss_scale_px=1.0, max_iterations=4)
    g = native.refine_intrinsics_arrays(p, **kw)
    r = oracle_lib.refine_intrinsics(p, **kw)
    for c, n in enumerate(counts):
        if n < 8:
            assert np.array_equal(g[c], p.camera_params[c])
        else:
            assert (np.abs(g[c] - r[c]) / np.maximum(np.abs(r[c]), 1.0)).max() <= 1e-6, (c, g[c], r[c])
