"""FP64 contractions on the tensor cores (gett_e64.cu) through jues_gemm: tile edges, K remainders, split K,
panels of A, the tiles handed back to the FP64 pipe, and the fall-back when no memory is left.

The reference is an exact product: each operand cut into integer parts whose float64 products and
sums are exact, added in extended precision.  The tensor-core form rounds the product once (2^-53), a
general alpha and a beta once more each, so three roundings bound the relative Frobenius error:
4 x 2^-53 is required.  Where tiles go back to the FP64 pipe the FMA loop's own bound
(K + 2) 2^-53 |A||B| is required element by element.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def exact(A, B):
    def parts(X, axis):
        m = np.max(np.abs(X), axis=axis, keepdims=True)
        m[m == 0] = 1.0
        e = np.ceil(np.log2(m))
        out, R = [], X.copy()
        for k in range(4):   # 4 x 17 bits
            s = 2.0 ** (e - 17 * (k + 1))
            h = np.rint(R / s)
            out.append((h, s.astype(np.longdouble)))
            R = R - h * s
        return out
    acc = np.zeros((A.shape[0], B.shape[1]), dtype=np.longdouble)
    for h, s in parts(A, 1):
        for g, t in parts(B, 0):
            acc += (h @ g).astype(np.longdouble) * (s * t)   # |h g| sums below 2^53: exact
    return acc


def rel(got, want):
    return np.linalg.norm((got - want).astype(float)) / np.linalg.norm(want.astype(float))


@pytest.mark.parametrize("M,N,K", [
    (1000, 70, 129),      # row maxima in their own pass just above one pack chunk
    (129, 1025, 128),     # one row past a tile, one column past a tile, K a whole pack chunk
    (2305, 49, 17),       # one K step and a remainder
    (5000, 33, 63),       # the last K step of a chunk partly filled
    (700, 300, 65),       # one K value in the second chunk
    (300, 300, 6401),     # few tiles, long K: K parts
    (128, 1024, 513),     # a single row tile
])
def test_gemm_fp64_is_rounded_once(M, N, K):
    from juesgpu import _lib
    rng = np.random.default_rng(M + N + K)
    A, B, C0 = rng.normal(size=(M, K)), rng.normal(size=(K, N)), rng.normal(size=(M, N))
    A[M // 2] = 0.0   # a zero row
    ex = exact(A, B)
    for ta, tb, al, be in ((0, 0, 1.0, 0.0), (1, 0, -0.5, 1.0), (0, 1, 0.3, 0.7), (1, 1, 2.0, 1.0)):
        got = _lib.gemm(np.asfortranarray(A.T if ta else A), np.asfortranarray(B.T if tb else B), C0, alpha=al,
                        beta=be, transA=bool(ta), transB=bool(tb), precision="fp64")
        want = np.longdouble(al) * ex + np.longdouble(be) * C0.astype(np.longdouble)
        assert rel(got, want) <= 4 * U
        if be == 0.0:
            assert np.all(got[M // 2] == 0.0)


def test_panels_of_a_long_operand():
    from juesgpu import _lib
    rng = np.random.default_rng(1)
    A, B = rng.normal(size=(190001, 90)), rng.normal(size=(90, 20))   # more rows than one panel of planes
    got = _lib.gemm(A, B, precision="fp64")
    rows = np.r_[0:300, 94000:101000, 189700:190001]
    assert rel(got[rows], exact(A[rows], B)) <= 4 * U
    assert np.abs(got - A @ B).max() <= 92 * U * (np.abs(A) @ np.abs(B)).max()


def test_special_and_graded_operands():
    from juesgpu import _lib
    rng = np.random.default_rng(2)
    A, B = rng.normal(size=(400, 300)), rng.normal(size=(300, 200))
    A[7, 3], A[200, 5], B[9, 50] = np.nan, np.inf, -np.inf
    A[100], A[150] = 0.0, 5e-310
    A[151] *= 1e200
    A[152] *= 1e-250
    with np.errstate(all="ignore"):
        want = A @ B
        got = _lib.gemm(A, B, precision="fp64")
        bound = 302 * U * (np.abs(A) @ np.abs(B))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(np.isinf(got), inf) and np.all(got[inf] == want[inf])
    f = np.isfinite(want)
    assert np.all(np.abs(got - want)[f] <= 2 * bound[f] + 1e-323)
    for span in (3, 12, 40):
        # rows of A fall and columns of B rise along K: each element's terms are alike, while the
        # largest elements of a row meet the smallest of a column
        g = 2.0 ** np.rint(np.linspace(0, -span, 300))
        x, y = rng.normal(size=(400, 300)), rng.normal(size=(300, 200))
        got = _lib.gemm(x * g, y / g[:, None], precision="fp64")
        assert np.all(np.abs((got - exact(x, y)).astype(float)) <= 302 * U * (np.abs(x) @ np.abs(y)))


def test_no_memory_for_planes_runs_on_the_fp64_pipe():
    from juesgpu import _lib
    ctx = _lib.Context(0)
    try:
        rng = np.random.default_rng(3)
        n = 640
        A, B = np.asfortranarray(rng.normal(size=(n, n))), np.asfortranarray(rng.normal(size=(n, n)))
        out = np.zeros((n, n), order="F")
        ctx.set_mem_limit(3 * 8 * n * n + (1 << 16))   # the three matrices and nothing else
        _lib.check(ctx.lib.jues_gemm(ctx.h, 0, 0, n, n, n, C.c_double(1.0), _lib.ptr(A), n, _lib.ptr(B), n,
                                     C.c_double(0.0), _lib.ptr(out), n, 0))
        assert np.all(np.abs((out - exact(A, B)).astype(float)) <= (n + 2) * U * (np.abs(A) @ np.abs(B)))
    finally:
        ctx.close()
