"""The batch's LU of windows whose Cholesky fails, all at once: one window and
many, a few unknowns and hundreds, windows that share a block's rows and
windows that take many blocks, beside windows that do not need it. A free
camera that sees nothing makes a window's system singular: its Cholesky fails
on a zero pivot, the LU skips the zero column and fails on it, and the damping
grows until the solve ends. Bars: those of the other degenerate windows in
test_gpu_batched.py (the oracle's iterations, cost 1e-6 relative)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native, scenes

pytestmark = pytest.mark.gpu

KW = dict(robust_loss=abi.LOSS_HUBER, max_iterations=6)


def _lonely(rng, images):
    p = scenes.local_window(rng, images, 25 * images)
    keep = p.obs_image != images // 2
    return p.copy(obs_image=p.obs_image[keep], obs_point=p.obs_point[keep], obs_xy=p.obs_xy[keep])


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sizes", [(3,), (4, 5, 4), (60,), (40, 3, 30, 6), (5,) * 60], ids=str)
def test_windows_that_reach_the_lu(oracle_lib, sizes, mixed):
    rng = np.random.default_rng(sum(sizes))
    wins = [_lonely(rng, m) for m in sizes] + [scenes.local_window(rng, 8, 200)]
    res = native.bundle_adjust_batched_arrays(
        wins, precision=abi.PRECISION_MIXED if mixed else abi.PRECISION_FP64, **KW)
    for k in {0, len(sizes) // 2, len(sizes) - 1, len(sizes)}:
        r = oracle_lib.bundle_adjust(wins[k], **KW)
        assert res[k].iterations_run == r.iterations_run
        assert abs(res[k].final_cost - r.final_cost) <= 1e-6 * r.final_cost
