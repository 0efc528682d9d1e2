"""The first results of a context: below 512 MB through the pair of 16 MB buffers, from there on through the 64 MB
slots, and both in turn."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# results of 16.8 MB (two fills), 96 MB (six) and 544 MB (nine slots)
@pytest.mark.parametrize("order", [(105000,), (600001, 105000), (600001, 3400000, 600001)])
def test_first_results(order):
    from juesgpu import _lib
    ctx = _lib.Context(0)
    rng = np.random.default_rng(len(order))
    B = np.asfortranarray(rng.integers(-8, 9, size=(3, 20)).astype(float))
    try:
        for rows in order:
            A = np.asfortranarray(rng.integers(-8, 9, size=(rows, 3)).astype(float))
            out = np.zeros((rows, 20), order="F")
            _lib.check(ctx.lib.jues_gemm(ctx.h, 0, 0, rows, 20, 3, C.c_double(1.0), _lib.ptr(A), rows, _lib.ptr(B), 3,
                                         C.c_double(0.0), _lib.ptr(out), rows, 0))
            assert np.array_equal(out, A @ B)   # small integers: exact
    finally:
        ctx.close()
