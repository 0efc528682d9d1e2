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
