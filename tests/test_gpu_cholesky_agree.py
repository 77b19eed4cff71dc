"""A pivot that fails while the trailing update of the block before it is still
at work on the other stream: the update's blocks must leave as a whole or not
at all, at any time the flag is set (tiles run in many waves here), and the
next factor is right.

Bar: a matrix that is not positive definite is reported, and the factor's
backward error (1e-14 of ||A||_F) as in test_gpu_dense_cholesky.py."""
import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


def test_pivots_that_fail_beside_the_update():
    n = 2500
    rng = np.random.default_rng(0)
    M = rng.standard_normal((n, n + 8))
    A = M @ M.T / n + 1e-2 * np.eye(n)
    for at in (64, 70, 127, 130, 200, 319, 640, 1000, 1791, 2111, 2430):
        keep = A[at, at]
        A[at, at] = -1.0
        for _ in range(3):
            with pytest.raises(native.SfmbaError, match="positive definite"):
                native.dense_cholesky(A, tensor_update=True)
        A[at, at] = keep
    L, _ = native.dense_cholesky(A, tensor_update=True)
    assert np.linalg.norm(A - L @ L.T) <= 1e-14 * np.linalg.norm(A)
