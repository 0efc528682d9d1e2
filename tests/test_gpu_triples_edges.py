"""(T) at the edges of the tiled energy kernel (8-wide virtual tiles) and of the stacked contractions (128 rows,
32 columns), and pair by pair when the stacked operands do not fit the memory limit.

Each term of the energy is a product of about ten roundings over sums of v + o products, and the
random signs cancel part of the sum: 1e-11 relative is required of FP64, 1e-6 of the split form (27-bit
operands).
"""
import ctypes as C

import numpy as np
import pytest

from oracle import triples

pytestmark = pytest.mark.gpu


def inputs(o, v, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(o, o, v, v))
    y = rng.normal(size=(v, o, v, o))
    z = rng.normal(size=(v, v, v, o))
    kw = dict(T1=0.1 * rng.normal(size=(o, v)), T2=x + x.transpose(1, 0, 3, 2), Vvvvo=z + z.transpose(1, 0, 2, 3),
              Vvooo=rng.normal(size=(v, o, o, o)), Vvovo=y + y.transpose(2, 3, 0, 1), fo=-1.0 - rng.random(o),
              fv=0.5 + rng.random(v))
    return {k: np.asfortranarray(a) for k, a in kw.items()}


@pytest.mark.parametrize("o,v", [(1, 1), (1, 9), (2, 7), (3, 16), (4, 17), (6, 11)])
def test_pT_edges(o, v):
    from juesgpu.CoupledCluster import PerturbativeTriples
    kw = inputs(o, v, 10 * o + v)
    want = triples.compute_pT(**kw)
    assert abs(PerturbativeTriples.compute_pT(**kw) - want) <= 1e-11 * abs(want)
    assert abs(PerturbativeTriples.compute_pT(precision="split", **kw) - want) <= 1e-6 * abs(want)


def test_pT_pair_by_pair_within_a_memory_limit():
    from juesgpu import _lib
    o, v = 4, 24
    kw = inputs(o, v, 5)
    words = sum(kw[k].size for k in ("T1", "T2", "Vvvvo", "Vvooo", "Vvovo", "fo", "fv"))
    ctx = _lib.Context(0)
    try:
        # the arrays, W of one pair and small tables; the stacked operands alone take 2.6 MB more
        ctx.set_mem_limit(8 * (words + v ** 3 * o) + (256 << 10))
        e = C.c_double()
        _lib.check(ctx.lib.jues_pT(ctx.h, *[_lib.ptr(kw[k]) for k in ("T1", "T2", "Vvvvo", "Vvooo", "Vvovo", "fo", "fv")],
                                   o, v, 0, C.byref(e)))
    finally:
        ctx.close()
    want = triples.compute_pT(**kw)
    assert abs(e.value - want) <= 1e-11 * abs(want)
