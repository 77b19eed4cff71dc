"""FP64 Schur reduction in chunks of a group's pairs, and the image right-hand
sides by one, two or eight warps: image pairs with fewer pairs than a chunk,
exactly one chunk, one more, and many; images with few and with many
observations; every block width. Whole solves against the oracle with the
bars of the other dense parity tests (same iterations; cost and parameters
1e-6: the sums differ from the oracle's by rounding only)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native, scenes

pytestmark = pytest.mark.gpu

MODELS = {6: None, 9: abi.SIMPLE_PINHOLE, 10: abi.SIMPLE_RADIAL, 11: abi.RADIAL, 14: abi.OPENCV}


@pytest.mark.parametrize("D", list(MODELS))
@pytest.mark.parametrize("images,points,views", [(3, 20, 3.0), (6, 32, 6.0), (6, 33, 6.0), (12, 500, 5.0), (5, 4000, 5.0)])
def test_chunk_ends_match_oracle(oracle_lib, D, images, points, views):
    model = abi.PINHOLE if MODELS[D] is None else MODELS[D]
    p = scenes.local_window(np.random.default_rng(100 * images + points), images, points, views=views, models=(model,))
    if MODELS[D] is None:
        p.fixed_cameras[:] = True
    assert p.block_width() == D
    kw = dict(robust_loss=abi.LOSS_HUBER, max_iterations=5)
    g = native.bundle_adjust_arrays(p, solver=abi.SOLVER_DENSE, **kw)
    r = oracle_lib.bundle_adjust(p, **kw)
    assert g.iterations_run == r.iterations_run
    assert abs(g.final_cost - r.final_cost) <= 1e-6 * r.final_cost
    for a, b in ((g.poses, r.poses), (g.points, r.points), (g.camera_params, r.camera_params)):
        assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
