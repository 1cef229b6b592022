"""fpp_dgemm_nt at the edges of its 256-row tiles of 64, 96 and 128 columns (the width that
fills the rounds of CTA pairs best), and past K = 65,536, where the group sums are converted
and combined as 64-bit integers of any size.

Bound: as in test_gpu_dgemm_digits.py, K (2^-54 + 2^-52) max|a_i| max|b_j| of the exact
product, and K 2^-53 of the same for the FP64 reference."""
import numpy as np
import pytest

from flare_pp_gb300._lib import check

pytestmark = pytest.mark.gpu


def dgemm(lib, A, B):
    (M, K), N = A.shape, B.shape[0]
    C = np.full((M, N), 7.0)
    check(lib.fpp_dgemm_nt(M, N, K, A.ctypes.data, K, B.ctypes.data, K, C.ctypes.data, N,
                           0, None))
    return C


@pytest.mark.parametrize("M,N,K", [
    (255, 63, 70), (256, 64, 64), (257, 65, 70), (256, 95, 70), (300, 97, 70), (513, 129, 70),
    (19456, 128, 70), (19456, 127, 65),  # 76 tiles of 128 columns: one round of 152 SMs
    (19456, 96, 70), (19455, 95, 70),    # of 96
    (9728, 129, 70), (9728, 191, 70), (9728, 192, 70), (9728, 193, 70)])
def test_edges_of_the_tiles(gpu_lib, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    C = dgemm(gpu_lib, A, B)
    scale = np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None]
    assert (np.abs(C - A @ B.T) <= K * (2.0 ** -54 + 2.0 ** -52 + 2.0 ** -53) * scale).all()


@pytest.mark.parametrize("M,N,K", [(3, 2, 65536), (2, 3, 65537), (130, 2, 70001)])
def test_long_sums(gpu_lib, M, N, K):
    """16-bit integers: every product and sum below 2^53, so the result is exact; and
    numbers of 53 bits against extended precision."""
    rng = np.random.default_rng(K)
    A = rng.integers(-2 ** 16, 2 ** 16, size=(M, K))
    B = rng.integers(-2 ** 16, 2 ** 16, size=(N, K))
    A[0], B[0] = 2 ** 16 - 1, 1 - 2 ** 16  # the largest sum
    C = dgemm(gpu_lib, A.astype(np.float64), B.astype(np.float64))
    np.testing.assert_array_equal(C, (A @ B.T).astype(np.float64))
    X, Y = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    C = dgemm(gpu_lib, X, Y)
    want = np.array([[(x.astype(np.longdouble) * y).sum() for y in Y] for x in X])
    bound = K * (2.0 ** -54 + 2.0 ** -52) * np.abs(X).max(1)[:, None] * np.abs(Y).max(1)[None]
    assert (np.abs(C - want) <= bound + 2.0 ** -52 * np.abs(C)).all()
