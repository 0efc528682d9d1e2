"""Small FP64 contractions: the edges of the small kernels' ranges against extended-precision products."""
import numpy as np
import pytest

from juesgpu import _lib

pytestmark = pytest.mark.gpu

# (M, N, K): one output pair and odd columns, lanes left over, the K table's edge (512), the lines of the
# dispatch (N = 8 / 9, K = 128 / 129, 4096 and 65536 outputs, K = 8192), K shorter than the lanes
SIZES = [(1, 2, 1), (33, 3, 7), (257, 5, 128), (257, 5, 129), (700, 8, 31), (70000, 2, 3),
         (9, 9, 1), (64, 64, 33), (64, 65, 33), (65, 64, 511), (65, 65, 512), (65, 65, 513),
         (256, 256, 16), (256, 257, 16), (455, 9, 8192), (456, 9, 8192),
         # staged tiles: K = 15 / 16, one and several chunks of K, 32768 outputs and one more row, thin tiles
         (100, 100, 15), (100, 100, 16), (90, 50, 385), (25, 400, 400), (128, 256, 20), (129, 256, 20), (3640, 9, 17)]


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_small_products(M, N, K, ta, tb):
    rng = np.random.default_rng(M * 7 + N * 3 + K)
    A = rng.normal(size=(K, M) if ta else (M, K))
    B = rng.normal(size=(N, K) if tb else (K, N))
    C0 = rng.normal(size=(M, N))
    a, b = (A.T if ta else A), (B.T if tb else B)
    # K products and their sum in any order, alpha, beta C and the last rounding: (K + 4) units of 2^-53 on
    # the sum of magnitudes; the reference in extended precision adds less than one more
    mag = 1.5 * (np.abs(a) @ np.abs(b)) + 0.5 * np.abs(C0)
    want = 1.5 * (a.astype(np.longdouble) @ b.astype(np.longdouble)) - 0.5 * C0.astype(np.longdouble)
    got = _lib.gemm(A, B, C=C0, alpha=1.5, beta=-0.5, transA=ta, transB=tb)
    assert np.all(np.abs(got - want) <= (K + 5) * 2.0 ** -53 * mag)


def test_small_products_nonfinite():
    A = np.ones((300, 10))
    B = np.ones((10, 5))
    A[3, 2], A[4, 9], A[299, 0] = np.nan, np.inf, -np.inf
    got = _lib.gemm(A, B)
    assert np.array_equal(np.isnan(got).any(axis=1), np.arange(300) == 3)
    assert np.all(got[4] == np.inf) and np.all(got[299] == -np.inf)
    assert np.all(np.delete(got, [3, 4, 299], axis=0) == 10.0)
