"""Results copied back through the staging ring (pageable arrays of 16 MB and more) and directly: sizes below
and above one ring slot (64 MB) and an array that is page-locked already, all equal to the plain product."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1000, 131073, 600001])   # 0.2 MB, 21 MB and 96 MB results
@pytest.mark.parametrize("pinned", [False, True])
def test_gemm_result_reaches_the_callers_array(rows, pinned):
    torch = pytest.importorskip("torch")
    from juesgpu import _lib
    ctx = _lib.context(0)
    rng = np.random.default_rng(rows)
    A = np.asfortranarray(rng.integers(-8, 9, size=(rows, 3)).astype(float))
    B = np.asfortranarray(rng.integers(-8, 9, size=(3, 20)).astype(float))
    if pinned:
        hold = torch.zeros(20, rows, dtype=torch.float64).pin_memory()
        out = hold.numpy().T
    else:
        out = np.zeros((rows, 20), order="F")
    _lib.check(ctx.lib.jues_gemm(ctx.h, 0, 0, rows, 20, 3, C.c_double(1.0), _lib.ptr(A), rows, _lib.ptr(B), 3,
                                 C.c_double(0.0), _lib.ptr(out), rows, 0))
    assert np.array_equal(out, A @ B)   # small integers: exact
