"""fpp_dgemm_nt at the edges of its digit planes: eight balanced 7-bit digits
of 55-bit fixed-point rows, level sums of at most 512 columns that reach the
FP32 significand, two halves of four levels, 128 x 128 tiles.

Bound: every operand entry is rounded to 2^-56 of 2^e (max |row| < 2^e), so an
entry errs by at most 2^-55 of its row's largest one, and the dropped digit pairs
(levels 8 and above, at most 7 pairs of 2^12 2^-68 per column, and the rest a
geometric tail) by 2^-52 of the product of the two row maxima.  Against exact
rational arithmetic:
    |C - A B^T| <= K (2 * 2^-55 + 2^-52 + 2^-110) max|a_i| max|b_j| + 2^-53 |C|
and exactly where every entry is a multiple of 2^-27 of its row's scale (28-bit
integers use the first four digits only)."""
import math
from fractions import Fraction

import numpy as np
import pytest

from flare_pp_gb300._lib import check

pytestmark = pytest.mark.gpu


def dgemm(lib, A, B):
    A = np.ascontiguousarray(A, dtype=np.float64)
    B = np.ascontiguousarray(B, dtype=np.float64)
    (M, K), N = A.shape, B.shape[0]
    C = np.full((M, N), 7.0)
    check(lib.fpp_dgemm_nt(M, N, K, A.ctypes.data, K, B.ctypes.data, K, C.ctypes.data, N,
                           0, None))
    return C


def exact(a, b):
    return sum(Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a, b))


@pytest.mark.parametrize("M,N,K", [(3, 5, 64), (129, 127, 65), (2, 130, 511), (2, 2, 512),
                                   (3, 2, 513), (2, 3, 1024), (2, 2, 1025), (257, 3, 576)])
def test_error_against_rational_arithmetic(gpu_lib, M, N, K):
    rng = np.random.default_rng(M + 10 * N + 100 * K)
    A = rng.normal(size=(M, K)) * 2.0 ** rng.integers(-40, 40, size=(M, 1))
    B = rng.normal(size=(N, K)) * 10.0 ** rng.uniform(-12, 0, size=(N, K))
    C = dgemm(gpu_lib, A, B)
    for i in sorted({0, M // 2, M - 1}):
        for j in sorted({0, N - 1}):
            x = exact(A[i], B[j])
            ra, rb = np.abs(A[i]).max(), np.abs(B[j]).max()
            bound = K * (2.0 ** -54 + 2.0 ** -52) * ra * rb + 2.0 ** -53 * abs(float(x))
            assert abs(float(Fraction(float(C[i, j])) - x)) <= bound, (i, j)


@pytest.mark.parametrize("K", [63, 512, 1536, 1600])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_largest_digits_of_one_sign(gpu_lib, K, sign):
    """Every digit at its bound (+64 then +63s and the like): the level sums
    reach 2^24 and must not lose a unit.  1 - 2^-53 and 0.5 + 0.25 + ... fill the
    digits; the product of equal rows is exact in rational arithmetic."""
    vals = np.array([1.0 - 2.0 ** -53, math.nextafter(0.5, 1.0), 63.0 / 64 + 63.0 / 8192,
                     sum(63.0 * 128.0 ** -(s + 1) for s in range(7))])
    A = np.tile(vals[:, None], (1, K))
    C = dgemm(gpu_lib, sign * A, A)
    for i, x in enumerate(vals):
        for j, y in enumerate(vals):
            want = K * Fraction(float(x)) * Fraction(float(y)) * int(sign)
            bound = K * (2.0 ** -54 + 2.0 ** -52) + 2.0 ** -53 * abs(float(want))
            assert abs(float(Fraction(float(C[i, j])) - want)) <= bound


def test_integers_of_28_bits_are_exact(gpu_lib):
    rng = np.random.default_rng(12)
    A = rng.integers(-2 ** 20, 2 ** 20, size=(140, 600)).astype(np.float64)
    B = rng.integers(-2 ** 20, 2 ** 20, size=(131, 600)).astype(np.float64)
    A[0], B[0] = 2 ** 20 - 1, 1 - 2 ** 20
    np.testing.assert_array_equal(dgemm(gpu_lib, A, B), A @ B.T)


def test_scales_and_non_finite_rows(gpu_lib):
    """Rows at the ends of the exponent range, subnormal rows, and rows with Inf
    or NaN, which come out NaN and leave the others alone."""
    rng = np.random.default_rng(13)
    A = rng.normal(size=(6, 70))
    B = rng.normal(size=(5, 70))
    ref = A @ B.T
    s = np.array([2.0 ** 1000, 2.0 ** -1000, 1.0, 1.0, 2.0 ** -500, 1.0])
    C = dgemm(gpu_lib, A * s[:, None], B)
    np.testing.assert_allclose(C / s[:, None], ref, rtol=0, atol=1e-13)
    tiny = np.full((1, 70), 3 * 2.0 ** -1074)
    big = np.full((1, 70), 2.0 ** 1000)
    assert dgemm(gpu_lib, tiny, big)[0, 0] == 70 * 3 * 2.0 ** -74
    A[2, 5], A[3, 69] = np.inf, np.nan
    B[4, 0] = -np.inf
    C = dgemm(gpu_lib, A, B)
    bad = np.zeros(C.shape, bool)
    bad[2:4] = bad[:, 4] = True
    assert np.isnan(C[bad]).all()
    np.testing.assert_allclose(C[~bad], ref[~bad], rtol=0, atol=1e-13)
