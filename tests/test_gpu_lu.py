"""The LU fallback where it succeeds (sfmba_dense_lu): systems that need real
pivoting (no usable diagonal, ties, permuted rows, tiny leading entries), from
one unknown to several hundred, the dense solver's kernels and the batch's,
windows of unequal size that share blocks or take many, and systems that are
singular, in the one-launch form and in that of a launch per column.

Bar: normwise backward error 4 n u g, u = 2^-53 and g the growth max|U| /
max|A| of LAPACK's factor with the same pivoting (Gaussian elimination's bound
is of this form with n^2; 4 n is above what it reaches). Every entry sees its
operations in the order of the swapping column loop, so both forms give the
same bits."""
import numpy as np
import pytest
import scipy.linalg

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


def _matrix(kind, n, rng):
    if kind == "indefinite":
        M = rng.standard_normal((n, n))
        return M + M.T
    if kind == "no_diagonal" and n > 1:  # [[0, B], [B^T, 0]], a random one for an odd n's middle
        h = n // 2
        A = np.zeros((n, n))
        A[n - h:, :h] = rng.standard_normal((h, h)) + 2.0 * np.eye(h)
        A[:h, n - h:] = A[n - h:, :h].T
        if n % 2:
            A[h, h] = 1.5
        return A
    if kind == "ties":  # rows of a permutation times signs, plus a few equal entries
        A = np.zeros((n, n))
        A[rng.permutation(n), np.arange(n)] = rng.choice([-1.0, 1.0], n)
        k = max(1, n // 8)
        A[:k, n - k:] += 0.5
        return A
    if kind == "permuted_rows":
        A = 0.1 * rng.standard_normal((n, n)) / np.sqrt(n) + np.eye(n)
        return A[rng.permutation(n)]
    A = rng.standard_normal((n, n))  # tiny leading entries
    A[: n // 2, : n // 2] *= 1e-200
    return A


KINDS = ["indefinite", "no_diagonal", "ties", "permuted_rows", "tiny_corner"]


def _check(A, x, b):
    n = len(b)
    assert x is not None
    U = scipy.linalg.lu(A)[2]
    growth = max(1.0, np.abs(U).max() / np.abs(A).max())
    back = np.abs(A @ x - b).max() / (np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max())
    assert back <= 4 * max(n, 4) * 2.0 ** -53 * growth, (n, back, growth)


@pytest.mark.parametrize("batched", [False, True], ids=["dense", "batch"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 31, 64, 65, 152, 153, 305, 607, 652])
@pytest.mark.parametrize("kind", KINDS)
def test_one_system(kind, n, batched):
    rng = np.random.default_rng(n)
    A, b = _matrix(kind, n, rng), rng.standard_normal(n)
    x = native.dense_lu([A], [b], batched=batched)[0]
    _check(A, x, b)
    assert np.array_equal(x, native.dense_lu([A], [b], batched=batched, by_columns=True)[0])


@pytest.mark.parametrize("sizes", [(1, 1), (333, 1, 7, 64, 40), (200, 201, 199, 3), tuple(range(1, 60)) * 3,
                                   (24,) * 700, (300,) * 24, (2000,) + (2, 3) * 500],
                         ids=["ones", "unequal", "large", "many", "small", "shared", "several_launches"])
def test_windows_of_a_batch(sizes):
    rng = np.random.default_rng(len(sizes))
    As = [_matrix(KINDS[k % len(KINDS)], n, rng) for k, n in enumerate(sizes)]
    bs = [rng.standard_normal(n) for n in sizes]
    xs = native.dense_lu(As, bs)
    for A, x, b in zip(As, xs, bs):
        _check(A, x, b)
    for x, y in zip(xs, native.dense_lu(As, bs, by_columns=True)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("by_columns", [False, True])
@pytest.mark.parametrize("batched", [False, True], ids=["dense", "batch"])
def test_singular_systems_are_told(batched, by_columns):
    rng = np.random.default_rng(5)
    zero_column = rng.standard_normal((90, 90))
    zero_column[:, 30] = 0.0
    same_rows = rng.integers(-3, 4, (4, 4)).astype(float) + 8.0 * np.eye(4)
    same_rows[3] = same_rows[1]
    for A in (np.zeros((1, 1)), zero_column, same_rows, np.zeros((70, 70))):
        good = _matrix("permuted_rows", 50, rng)
        b = rng.standard_normal(len(A))
        if not batched:
            assert native.dense_lu([A], [b], batched=False, by_columns=by_columns) == [None]
            continue
        x = native.dense_lu([good, A, good], [np.ones(50), b, np.arange(50.0)], by_columns=by_columns)
        assert x[1] is None
        _check(good, x[0], np.ones(50))
        _check(good, x[2], np.arange(50.0))
