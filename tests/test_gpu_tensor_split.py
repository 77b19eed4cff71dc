"""Digits of the tensor-core update at the ends of the exponent range: rows of
very different scale, blocks of zeros, matrices whose factor lies near the
smallest and the largest normal numbers.

Bar: test_gpu_dense_cholesky.py's backward error (1e-14 of ||A||_F) of the
matrix brought back to unit scale by powers of two, which is exact."""
import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-960, -300, 0, 300, 960])
@pytest.mark.parametrize("zeros", [False, True], ids=["dense", "zero-blocks"])
def test_split_over_the_exponent_range(power, zeros):
    n = 193
    rng = np.random.default_rng(abs(power))
    M = rng.standard_normal((n, n + 8))
    A = M @ M.T / n + 1e-2 * np.eye(n)
    if zeros:  # panel rows of zeros below the first two blocks
        A[100:, :100] = 0.0
        A[:100, 100:] = 0.0
    d = 2.0 ** rng.integers(-12, 13, n)
    L, _ = native.dense_cholesky(np.ldexp(d[:, None] * A * d[None, :], power), tensor_update=True)
    L = np.ldexp(L, -power // 2) / d[:, None]
    assert np.linalg.norm(A - L @ L.T) <= 1e-14 * np.linalg.norm(A)
