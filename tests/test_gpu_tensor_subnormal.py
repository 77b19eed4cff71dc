"""Panel rows of subnormal numbers in the tensor-core update: their digits are
exact like any other row's.

Bar: a subnormal result is a multiple of 2^-1074 and every operation on one
rounds by half of that. An entry sees 64 multiply-adds a panel (or one
conversion) in two panels, then the product with a block's inverse (64 more)
whose rows here sum to less than 2: 512 x 2^-1074 covers both factors' errors.
The entries themselves are some 1e13 times 2^-1074."""
import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


def test_subnormal_rows():
    rng = np.random.default_rng(3)
    n, m = 256, 128
    A = np.eye(n)
    M = rng.standard_normal((m, m)) / 40.0
    A[:m, :m] += M @ M.T
    A[m:, :m] = 1e-310 * rng.standard_normal((n - m, m))
    A[:m, m:] = A[m:, :m].T
    Lf, _ = native.dense_cholesky(A, tensor_update=False)
    Lt, _ = native.dense_cholesky(A, tensor_update=True)
    assert np.abs(Lf[m:, 64:m]).max() > 1e-310
    assert np.abs(Lt[m:, :m] - Lf[m:, :m]).max() <= 512 * 2.0 ** -1074
    assert np.abs(Lt[:m] - Lf[:m]).max() <= 1e-14
