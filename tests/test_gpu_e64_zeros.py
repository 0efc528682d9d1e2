"""FP64 contractions on the tensor cores with the zero pattern of symmetry: rows, columns and K belong to irreducible
representations in turn, and only those of one representation meet.

Exact zeros must not send anything back to the FP64 pipe.  The digit form rounds a result once, so nearly every
element is the exact product rounded to nearest; a sum of a dozen and more FMAs, each rounded, is that for about half
of the elements.  So at least nine tenths of the elements are required to be the rounded exact product.
"""
import numpy as np
import pytest

from test_gpu_e64 import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("irreps", [2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(3000, 40, 100), (700, 260, 200), (130, 70, 9000), (400, 300, 56)])
def test_symmetry_zeros_stay_on_the_tensor_cores(M, N, K, irreps):
    from juesgpu import _lib
    rng = np.random.default_rng(M + K + irreps)
    m, n, k = (np.arange(x) % irreps for x in (M, N, K))
    A = rng.normal(size=(M, K)) * (m[:, None] == k[None, :])
    B = rng.normal(size=(K, N)) * (k[:, None] == n[None, :])
    want = exact(A, B)
    for got in (_lib.gemm(A, B, precision="fp64"),
                _lib.gemm(np.asfortranarray(B.T), np.asfortranarray(A.T), precision="fp64").T):
        live = m[:, None] == n[None, :]
        assert np.all(got[~live] == 0.0)
        assert np.mean(got[live] == want[live].astype(float)) >= 0.9
