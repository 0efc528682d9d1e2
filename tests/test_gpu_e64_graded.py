"""FP64 contractions on the tensor cores whose rows and columns mix magnitudes: every element keeps the bound of an
FMA loop, (K + 5) 2^-53 |A||B|, also where the large elements of a row meet zeros of the column.

The operands are A = [x1 | s x2] and B = [y1; y2] with s = 1 in some rows, s tiny in others, and y1 = 0 in some
columns, in patterns finer than any tile.  The reference adds the two halves' exact products.
"""
import numpy as np
import pytest

from test_gpu_e64 import exact

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def operands(M, N, K, s, every, rng):
    h = K // 2
    x, y = rng.normal(size=(M, K)), rng.normal(size=(K, N))
    low, cut = np.arange(M) % every == 0, np.arange(N) % every == 1
    g = np.where(low, s, 1.0)[:, None]
    keep = np.where(cut, 0.0, 1.0)[None, :]
    A, B = x.copy(), y.copy()
    A[:, h:] *= g
    B[:h] *= keep
    want = exact(x[:, :h], y[:h]) * keep + exact(x[:, h:], y[h:]) * g.astype(np.longdouble)
    return A, B, want


@pytest.mark.parametrize("bits", [6, 10, 20, 30, 80])
@pytest.mark.parametrize("M,N,K,every", [
    (600, 200, 50, 2),      # K in one plane width; rows and columns in turn
    (700, 130, 100, 5),     # the other width
    (300, 260, 400, 8),     # row maxima in their own pass; one row of eight in a thread's columns
    (260, 129, 4000, 2),    # K parts
    (260, 129, 9000, 32),   # parts folded in groups; one column of a tile
])
def test_mixed_grading_keeps_each_element(M, N, K, every, bits):
    from juesgpu import _lib
    rng = np.random.default_rng(M + N + K + bits)
    A, B, want = operands(M, N, K, 2.0 ** -bits, every, rng)
    bound = (K + 5) * U * (np.abs(A) @ np.abs(B))
    got = _lib.gemm(A, B, precision="fp64")
    assert np.all(np.abs((got - want).astype(float)) <= bound)
    # the roles of the operands traded
    got = _lib.gemm(np.asfortranarray(B.T), np.asfortranarray(A.T), precision="fp64")
    assert np.all(np.abs((got.T - want).astype(float)) <= bound)


@pytest.mark.parametrize("bits", [12, 40, 90])
def test_only_small_elements_meet(bits):
    # A = [x1 | s x2 | 0], B = [0; s y2; y3] in every third row and column: the results are s^2 x2.y2
    from juesgpu import _lib
    rng = np.random.default_rng(bits)
    M, N, K, h = 500, 270, 192, 64
    x, y, s = rng.normal(size=(M, K)), rng.normal(size=(K, N)), 2.0 ** -bits
    A, B = x.copy(), y.copy()
    A[::3, h:2 * h] *= s
    A[::3, 2 * h:] = 0.0
    B[h:2 * h, 1::3] *= s
    B[:h, 1::3] = 0.0
    want = exact(x, y)
    want[::3] = exact(x[::3, :h], y[:h]) + exact(x[::3, h:2 * h], y[h:2 * h]) * np.longdouble(s)
    want[:, 1::3] = exact(x[:, h:2 * h], y[h:2 * h, 1::3]) * np.longdouble(s) + exact(x[:, 2 * h:], y[2 * h:, 1::3])
    want[::3, 1::3] = exact(x[::3, h:2 * h], y[h:2 * h, 1::3]) * np.longdouble(s) * np.longdouble(s)
    got = _lib.gemm(A, B, precision="fp64")
    assert np.all(np.abs((got - want).astype(float)) <= (K + 5) * U * (np.abs(A) @ np.abs(B)))


def test_every_tile_left_out():
    # all rows graded: far more tiles than the short and middle lists hold
    from juesgpu import _lib
    rng = np.random.default_rng(7)
    A, B, want = operands(9000, 400, 60, 2.0 ** -40, 1, rng)
    B[:30, 1::2] = 0.0
    x = A[:, 30:]
    want[:, 1::2] = exact(x * 2.0 ** 40, B[30:, 1::2]) * np.longdouble(2.0 ** -40)
    got = _lib.gemm(A, B, precision="fp64")
    assert np.all(np.abs((got - want).astype(float)) <= 65 * U * (np.abs(A) @ np.abs(B)))


# few elements of a half tile below the line (listed one by one), with every way of storing the others; 41 rows apart,
# so that pieces of both column groups and of the last, short row and column tiles are among them
@pytest.mark.parametrize("M,N,K", [(1300, 83, 100), (400, 150, 300), (200, 70, 6000)])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-2.0, 1.0), (0.3, -0.7)])
@pytest.mark.parametrize("transB", [False, True])
def test_few_elements_left_out(M, N, K, alpha, beta, transB):
    from juesgpu import _lib
    rng = np.random.default_rng(M + N + K)
    A, B, want = operands(M, N, K, 2.0 ** -40, 41, rng)
    A[-1], want[-1] = 0.0, 0.0
    C0 = rng.normal(size=(M, N))
    got = _lib.gemm(A, np.asfortranarray(B.T) if transB else B, C=C0, alpha=alpha, beta=beta, transB=transB,
                    precision="fp64")
    full = np.longdouble(alpha) * want + np.longdouble(beta) * C0.astype(np.longdouble)
    mag = abs(alpha) * (np.abs(A) @ np.abs(B)) + abs(beta) * np.abs(C0)
    assert np.all(np.abs((got - full).astype(float)) <= (K + 5) * U * mag)
    # and with beta = 0 the small elements keep their own bound beside the large ones
    if beta == 0.0:
        low = want[::41, 1::41]
        assert np.all(np.abs((got[::41, 1::41] - alpha * low).astype(float)) <= (K + 5) * U * mag[::41, 1::41])
