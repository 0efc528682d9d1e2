"""Tensor-core FP64 contractions with many K parts, and with tiles left to the FP64 pipe in short and longer lists."""
import numpy as np
import pytest

from juesgpu import _lib

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def check(A, B, C0):
    K = A.shape[1]
    got = _lib.gemm(A, B, C=C0, alpha=-1.5, beta=0.5)
    want = -1.5 * (A.astype(np.longdouble) @ B.astype(np.longdouble)) + 0.5 * C0.astype(np.longdouble)
    mag = 1.5 * (np.abs(A) @ np.abs(B)) + 0.5 * np.abs(C0)
    # K products and their sum in any order, alpha, beta C and the last rounding
    assert np.all(np.abs(got - want) <= (K + 5) * U * mag)


# one tile and few, a number of parts that is no multiple of the group of eight
@pytest.mark.parametrize("M,N,K", [(13, 17, 40000), (100, 40, 4100), (129, 33, 2000), (128, 32, 8192)])
def test_many_parts(M, N, K):
    rng = np.random.default_rng(M + N + K)
    check(rng.normal(size=(M, K)), rng.normal(size=(K, N)), rng.normal(size=(M, N)))


# rows orthogonal to a 16-wide range of columns: their results nearly vanish and the tile is left out
@pytest.mark.parametrize("tiles", [1, 16, 17, 44])
@pytest.mark.parametrize("transB", [False, True])
def test_left_out_tiles(tiles, transB):
    M, N, K = 1300, 51, 130   # 11 x 4 tiles, the last ones 20 rows and 3 columns
    rng = np.random.default_rng(tiles)
    A = rng.normal(size=(M, K))
    B = np.ascontiguousarray(rng.normal(size=(N, K))).T if transB else rng.normal(size=(K, N))
    for t in rng.permutation(44)[:tiles]:
        r, c = 128 * (t % 11) + 3, 16 * (t // 11)
        q, _ = np.linalg.qr(B[:, c:c + 16])
        A[r] -= q @ (q.T @ A[r])
    check(A, B, rng.normal(size=(M, N)))
