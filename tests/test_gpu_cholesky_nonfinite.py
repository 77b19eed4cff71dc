"""NaN and infinity in a panel that the tensor-core update splits (below the
diagonal, where no pivot meets them directly): the row's own diagonal entry
must fail, as it does with FP64 updates. Bar: the matrix is reported as not
positive definite by both forms, and the next factor is right (1e-14 of
||A||_F, as in test_gpu_dense_cholesky.py)."""
import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor", [False, True], ids=["fma", "tensor"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [(64, 63), (130, 5), (130, 70), (199, 0), (199, 130), (199, 198), (70, 65)], ids=str)
def test_nonfinite_entry_of_a_panel(at, value, tensor):
    n = 200
    rng = np.random.default_rng(1)
    M = rng.standard_normal((n, n + 8))
    A = M @ M.T / n + 1e-2 * np.eye(n)
    B = A.copy()
    B[at] = B[at[::-1]] = value
    with pytest.raises(native.SfmbaError, match="positive definite"):
        native.dense_cholesky(B, tensor_update=tensor)
    L, _ = native.dense_cholesky(A, tensor_update=tensor)
    assert np.linalg.norm(A - L @ L.T) <= 1e-14 * np.linalg.norm(A)
