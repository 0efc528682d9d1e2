"""CCD's FP64 sweeps with the ladders folded over pairs, against the same sweeps unfolded."""
import re

import numpy as np
import pytest

from juesgpu import _lib
from juesgpu.CoupledCluster import CCSession
from juesgpu.synthetic import make_system

pytestmark = pytest.mark.gpu


def in_use(ctx):
    """Bytes allocated, as a refusal reports them."""
    ctx.set_mem_limit(1)
    with pytest.raises(_lib.JuESError) as e:
        _lib.gemm(np.ones((64, 64)), np.ones((64, 64)))
    ctx.set_mem_limit(0)
    return int(re.search(r"(\d+) in use", str(e.value)).group(1))


def solve(w, room):
    ctx = _lib.context(0)
    s = CCSession(0, w, maxit=6, r_conv=0.0)
    try:
        if room:
            ctx.set_mem_limit(in_use(ctx) + room)
        ctx.set_profiling(True)
        ctx.profile_reset()
        s.iterate(6)
        return s.energy(), s.amplitudes()[1], ctx.profile("pair_fold")[1]
    finally:
        ctx.set_profiling(False)
        ctx.set_mem_limit(0)
        s.close()


# just beyond the line (o^2 v^4 = 3.5e9): pair counts that are no multiples of a tile, few pairs
@pytest.mark.parametrize("n,o", [(75, 20), (76, 19), (100, 7)])
def test_folded_against_unfolded(n, o):
    w = make_system(n, o, 3 * n, seed=n + o).wfn()
    e1, t1, folds = solve(w, 0)
    # the unfolded sweeps' own arrays fit; the folded weights would not leave room for all that may still come
    e0, t0, none = solve(w, 24 * (n - o) ** 4)
    assert folds > 0 and none == 0
    # a sweep's ladder sums carry at most 2 v^2 + 2 units of 2^-53 of their magnitudes in either form
    tol = 20 * 2 * (n - o) ** 2 * 2.0 ** -53
    assert abs(e1 - e0) <= tol * abs(e0)
    assert np.abs(t1 - t0).max() <= tol * np.abs(t0).max()
