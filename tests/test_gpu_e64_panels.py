"""FP64 contractions whose digit planes go through panels: the results do not depend on the panels."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# planes of 188 MB (rows past a panel's edge, K in one pack block and in several); room for 188 MB, for one
# 128 MB panel, and for no planes at all (the FP64 pipe)
@pytest.mark.parametrize("M,N,K", [(60001, 20, 215), (119000, 33, 100)])
@pytest.mark.parametrize("transA", [0, 1])
def test_panels_under_a_memory_limit(M, N, K, transA):
    from juesgpu import _lib
    rng = np.random.default_rng(M + N + K)
    A = np.asfortranarray(rng.normal(size=(K, M) if transA else (M, K)))
    B = np.asfortranarray(rng.normal(size=(K, N)))
    operands = 8 * (M * K + K * N + M * N)
    ctx = _lib.Context(0)
    outs = []
    try:
        for room in (260 << 20, 150 << 20, 1 << 16):
            out = np.zeros((M, N), order="F")
            ctx.set_mem_limit(operands + room)
            _lib.check(ctx.lib.jues_gemm(ctx.h, transA, 0, M, N, K, C.c_double(1.0), _lib.ptr(A), A.shape[0],
                                         _lib.ptr(B), K, C.c_double(0.0), _lib.ptr(out), M, 0))
            outs.append(out)
    finally:
        ctx.close()
    assert np.array_equal(outs[0], outs[1])
    # the two forms differ by no more than both their bounds: K + 2 units of 2^-53 on the sum of magnitudes
    a = A.T if transA else A
    assert np.all(np.abs(outs[0] - outs[2]) <= 2 * (K + 2) * 2.0 ** -53 * (np.abs(a) @ np.abs(B)))


def test_panel_edges_against_exact_products():
    # planes of 274 MB and room for one panel of 128 MB: three panels, the rows on both sides of each edge exact but
    # for one rounding of the result (and 2^-61 of its row's and column's norms)
    from juesgpu import _lib
    from test_gpu_e64 import U, exact, rel
    M, N, K = 190001, 20, 90
    rng = np.random.default_rng(11)
    A, B = np.asfortranarray(rng.normal(size=(M, K))), np.asfortranarray(rng.normal(size=(K, N)))
    out = np.zeros((M, N), order="F")
    ctx = _lib.Context(0)
    try:
        ctx.set_mem_limit(8 * (M * K + K * N + M * N) + (150 << 20))
        _lib.check(ctx.lib.jues_gemm(ctx.h, 0, 0, M, N, K, C.c_double(1.0), _lib.ptr(A), M, _lib.ptr(B), K,
                                     C.c_double(0.0), _lib.ptr(out), M, 0))
    finally:
        ctx.close()
    # 2^26 words of 2 bytes, 96 padded K values in seven planes and half a word for the magnitude, whole row tiles
    prow = 2 ** 26 * 2 // (15 * 96) // 128 * 128
    assert prow < M // 2
    for edge in (prow, 2 * prow):
        rows = slice(edge - 200, edge + 200)
        assert rel(out[rows], exact(A[rows], B)) <= 4 * U
    rows = np.r_[0:200, M - 200:M]
    assert rel(out[rows], exact(A[rows], B)) <= 4 * U
