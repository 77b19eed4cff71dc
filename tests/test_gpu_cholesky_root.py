"""The pivots' square roots and reciprocals: an arrow matrix, diagonal but for
its last row x, has L_ii = sqrt(d_i) and L_ni = x_i (1 / sqrt(d_i)), one
rounding each, at every place of a diagonal block and in the panel. Bar: the
bits of numpy's correctly rounded root, division and product."""
import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


def _pivots(kind, rng, n):
    m = 1.0 + rng.random(n)
    if kind == "any exponent":
        return np.ldexp(m, rng.integers(-1000, 1000, n))
    if kind == "both parities":
        return np.ldexp(m, rng.integers(-2, 3, n))
    if kind == "squares and beside":  # roots that are exact, and those that end near one
        return np.nextafter(m.astype(np.float32).astype(np.float64) ** 2, rng.choice([0.0, 2.0, 9.0], n))
    if kind == "roots near ties":
        return np.nextafter(m * m, rng.choice([0.0, 9.0], n))
    if kind == "ends of a binade":
        return np.ldexp(1.0 + rng.integers(-8, 8, n) * 2.0**-52, rng.integers(-3, 4, n))
    return np.ldexp(rng.random(n) + 2.0**-20, -1040)  # subnormal


@pytest.mark.parametrize("n", [64, 1000])
@pytest.mark.parametrize("kind", ["any exponent", "both parities", "squares and beside", "roots near ties",
                                  "ends of a binade", "subnormal"])
def test_pivots_are_rounded_once(n, kind):
    rng = np.random.default_rng(n)
    d = _pivots(kind, rng, n - 1)
    root = np.sqrt(d)
    x = root * rng.uniform(-1.0, 1.0, n - 1)
    A = np.zeros((n, n))
    A[np.arange(n - 1), np.arange(n - 1)] = d
    A[-1, :-1] = A[:-1, -1] = x
    A[-1, -1] = 2.0 * n
    L, _ = native.dense_cholesky(A)
    assert np.array_equal(np.diag(L)[:-1], root)
    assert np.array_equal(L[-1, :-1], x * (1.0 / root))
