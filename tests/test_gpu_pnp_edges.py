"""PnP registration where the FP32 filter of its inlier test and its null
vectors could go wrong: worlds far from the origin and of large and small
scale (the filter's bounds and the conditioning of the DLT follow them),
points behind and next to the camera plane, a threshold that a residual meets
exactly, exact (singular) and noisy systems, the fewest correspondences and
batches around a block's size, against the oracle.

Bars: those of test_gpu_pnp.py (same registered images, iterations and inlier
masks, poses 1e-9), the translation relative to the world's size."""
import numpy as np
import pytest

from sfmtory_gb300 import native, scenes
from sfmtory_gb300.problem import quat_to_matrix

pytestmark = pytest.mark.gpu


def _same(oracle_lib, Xs, uvs, thr, iterations=300):
    got = native.pnp_ransac_batched(Xs, uvs, thr, iterations)
    for k in range(len(Xs)):
        ref = oracle_lib.pnp_ransac(Xs[k], uvs[k], thr, iterations)
        assert (got[k] is None) == (ref is None), k
        if ref is None:
            continue
        assert got[k][2] == ref[2], (k, got[k][2], ref[2])
        assert np.array_equal(got[k][1], ref[1]), k
        a, b = got[k][0], ref[0]
        assert min(np.abs(a[:4] - b[:4]).max(), np.abs(a[:4] + b[:4]).max()) <= 1e-9, k
        assert np.abs(a[4:] - b[4:]).max() <= 1e-9 * max(1.0, np.abs(b[4:]).max()), k


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3])
@pytest.mark.parametrize("outliers", [0.0, 0.4])
def test_world_scales(oracle_lib, scale, outliers):
    _, Xs, uvs, thr = scenes.pnp_batch(5, num_images=9, n_min=40, n_max=300, outlier_frac=outliers)
    _same(oracle_lib, [X * scale for X in Xs], uvs, thr)


def test_points_behind_and_beside_the_camera(oracle_lib):
    poses, Xs, uvs, thr = scenes.pnp_batch(6, num_images=5, n_min=60, n_max=200, outlier_frac=0.2)
    rng = np.random.default_rng(1)
    out = []
    for pose, X in zip(poses, Xs):
        R = quat_to_matrix(pose[:4])
        pc = X @ R.T + pose[4:]
        some = rng.choice(len(X), 12, replace=False)
        pc[some[:4], 2] *= -1.0
        pc[some[4:8], 2] = 0.0
        pc[some[8:], 2] = 1e-9
        out.append((pc - pose[4:]) @ R)
    _same(oracle_lib, out, uvs, thr)


def test_threshold_met_exactly(oracle_lib):
    """An identity camera and dyadic coordinates: some residuals equal the
    threshold, which does not count as an inlier."""
    rng = np.random.default_rng(2)
    pc = np.concatenate([rng.integers(-64, 65, (120, 2)) / 64.0, rng.integers(2, 6, (120, 1)).astype(float)], 1)
    uv = pc[:, :2] / pc[:, 2:]
    uv[:40, 0] += 2.0 ** -7
    uv[40:60, 1] -= 2.0 ** -7
    _same(oracle_lib, [pc], [uv], 2.0 ** -7)


@pytest.mark.parametrize("images,n", [(1, 6), (3, 7), (2, 33), (130, 12)])
def test_fewest_correspondences_and_batch_sizes(oracle_lib, images, n):
    _, Xs, uvs, thr = scenes.pnp_batch(images + n, num_images=images, n_min=n, n_max=n, outlier_frac=0.0)
    _same(oracle_lib, Xs, uvs, thr, iterations=40)
