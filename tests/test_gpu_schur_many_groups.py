"""FP64 Schur reduction where the image pairs alone fill the GPU (1830 of them,
of up to 150 common points): their chunks are launched longest first, and pairs
of at most two rounds are not cut. A whole solve against the oracle, with the
bars of the other dense parity tests (same iterations; cost and parameters
1e-6)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [60, 300])
def test_many_image_pairs_match_oracle(oracle_lib, points):
    p = scenes.local_window(np.random.default_rng(points), 60, points, views=30.0, models=(abi.SIMPLE_RADIAL,))
    kw = dict(robust_loss=abi.LOSS_HUBER, max_iterations=4)
    g = native.bundle_adjust_arrays(p, solver=abi.SOLVER_DENSE, **kw)
    r = oracle_lib.bundle_adjust(p, **kw)
    assert g.iterations_run == r.iterations_run
    assert abs(g.final_cost - r.final_cost) <= 1e-6 * r.final_cost
    for a, b in ((g.poses, r.poses), (g.points, r.points), (g.camera_params, r.camera_params)):
        assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
