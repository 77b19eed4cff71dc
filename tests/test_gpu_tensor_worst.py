"""The tensor-core update where its bounds are largest: panel rows whose digits
are all 255 or close to it, all of one sign, against exact rationals.

The leading 64 x 64 block is the identity, so the panel is the matrix's own
rows, and column 64 of the next block, whose pivot is exactly 4, shows the
updated entries as D / 2. With s = 1 the scale of both rows, an entry's error
is at most: 2^-47 (the update, below 64, rounded to 53 bits), 2^-47.3 (the
products of weight 9 and more that are left out), the roundings of the FP32
sums past 2^24 in the group of weight 6 (its last four of 20 instructions, a
unit of 2 each at most: 2^-45), 2^-48 (the 64-bit sum rounded to 53 bits), 2^-54
(the other groups): below 2^-44. The bound of 64 multiply-adds in FP64 is
2^-41."""
from fractions import Fraction

import numpy as np
import pytest

from sfmtory_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ones", "mixed", "low", "random"])
def test_digits_close_to_255(kind):
    n = 128
    rng = np.random.default_rng(len(kind))
    bits = np.full((64, 64), (1 << 53) - 1, dtype=np.int64)
    if kind == "mixed":  # digits 254 and 255
        for at in range(0, 48, 8):
            bits -= rng.integers(0, 2, bits.shape) << (45 - at)
    elif kind == "low":  # the lowest digits move the group sums past 2^24 by odd amounts
        bits -= rng.integers(0, 1 << 13, bits.shape)
    elif kind == "random":
        bits = rng.integers(1 << 52, 1 << 53, bits.shape)
    P = np.ldexp(bits.astype(np.float64), -53)
    exact = [sum(Fraction(int(bits[r, t]) * int(bits[0, t]), 1 << 106) for t in range(64)) for r in range(64)]
    A = np.eye(n)
    A[64:, :64] = P
    A[:64, 64:] = P.T
    A[64:, 64:] = 1e4 * np.eye(64)
    for r in range(64):
        A[64 + r, 64] = A[64, 64 + r] = float(exact[r])
    A[64, 64] = float(exact[0]) + 4.0
    L, _ = native.dense_cholesky(A, tensor_update=True)
    assert np.array_equal(L[:64, :64], np.eye(64)) and np.array_equal(L[64:, :64], P)
    worst = 0.0
    for r in range(1, 64):
        D = Fraction(float(L[64 + r, 64])) * Fraction(float(L[64, 64]))
        worst = max(worst, abs(float(Fraction(float(A[64 + r, 64])) - D - exact[r])))
    # the pivot's own entry carries the same error: relative to D, which is below 2^-45, it does not show
    assert worst <= 2.0 ** -44, worst * 2.0 ** 47
