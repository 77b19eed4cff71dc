"""The blocked Cholesky and the dense solve where their blocks end: diagonal
blocks of 1 to 64 columns, panels of 8 rows, update tiles of 16 and 32 (and
the sizes that switch between them), pivots that fail at every kind of place,
and solves of one and of many 64-wide blocks.

Bars: the factor's backward error (1e-14 of ||A||_F) and its difference from
LAPACK's (100 ulp times the condition number), as in
test_gpu_dense_cholesky.py; whole solves against the oracle with the bars of
the other dense parity tests (same iterations, cost and parameters 1e-6)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native, scenes

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    rng = np.random.default_rng(seed)
    M = rng.standard_normal((n, n + 8))
    return M @ M.T / n + 1e-2 * np.eye(n)


@pytest.mark.parametrize("tensor", [False, True], ids=["fma", "tensor"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 71, 72, 73, 79, 80, 81, 95, 96, 97, 128, 129, 200,
                               600, 700])
def test_factor_at_block_ends(n, tensor):
    A = _spd(n, seed=n)
    L, _ = native.dense_cholesky(A, tensor_update=tensor)
    assert np.linalg.norm(A - L @ L.T) <= 1e-14 * np.linalg.norm(A)
    Ln = np.linalg.cholesky(A)
    assert np.abs(L - Ln).max() <= max(1e-14 * np.linalg.cond(A), 1e-13) * np.abs(Ln).max()


@pytest.mark.parametrize("at", [0, 1, 2, 31, 32, 63, 64, 65, 127, 149])
@pytest.mark.parametrize("value", [-1.0, 0.0, np.nan])
def test_failed_pivot_is_reported(at, value):
    A = _spd(150, seed=7)
    A[at, at] = value
    if value == 0.0:
        A[at, :] = A[:, at] = 0.0
    with pytest.raises(native.SfmbaError, match="positive definite"):
        native.dense_cholesky(A)


@pytest.mark.parametrize("images", [2, 8, 9, 17, 60])
def test_solve_of_one_and_many_blocks(oracle_lib, images):
    p = scenes.local_window(np.random.default_rng(images), images, 40 * images, views=3.0, models=(abi.OPENCV,))
    kw = dict(robust_loss=abi.LOSS_NONE, max_iterations=6)
    g = native.bundle_adjust_arrays(p, solver=abi.SOLVER_DENSE, **kw)
    r = oracle_lib.bundle_adjust(p, **kw)
    assert g.iterations_run == r.iterations_run
    assert abs(g.final_cost - r.final_cost) <= 1e-6 * r.final_cost
    for a, b in ((g.poses, r.poses), (g.points, r.points), (g.camera_params, r.camera_params)):
        assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
