"""Bounded waits of the blocked Cholesky that give up (test aid: at once): of the
blocks that follow a diagonal block's columns, of one block of 64 columns, of
blocks with and without a second half, of many; of the tensor-core tiles, one
and many. They are an internal error, not a matrix that is not positive
definite; the kernels end, and the next factor is right (1e-14 of ||A||_F, as
in test_gpu_dense_cholesky.py)."""
import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor,tiles", [(False, False), (True, False), (True, True)],
                         ids=["columns-fma", "columns-tensor", "tiles"])
@pytest.mark.parametrize("n", [1, 20, 32, 33, 64, 65, 150, 1100])
def test_a_wait_that_gives_up_is_an_internal_error(n, tensor, tiles):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n + 8))
    A = M @ M.T / n + 1e-2 * np.eye(n)
    if not tiles or n > 64:  # one block of columns has no tiles
        with pytest.raises(native.SfmbaError, match="bounded wait") as e:
            native.dense_cholesky_give_up(A, tensor, tiles)
        assert e.value.status != 1  # INVALID_ARGUMENT
    L, _ = native.dense_cholesky(A, tensor_update=tensor)
    assert np.linalg.norm(A - L @ L.T) <= 1e-14 * np.linalg.norm(A)
