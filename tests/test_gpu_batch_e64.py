"""The batched FP64 form on the tensor cores: stages large enough for the grouped digit planes (K <= 64 in one
plane width and K <= 128 in the other), the K-split dE/dC stage, and the kept first quarter, against the
single-system adjoint (1e-13 of the largest entry: sums of at most 70^3 products rounded once per stage)."""
import numpy as np
import pytest

from juesgpu.synthetic import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [(30, 6), (41, 8), (64, 13), (17, 3), (64, 40)],    # nocc > nvir in one: no kept quarter there
    [(33, 7), (70, 12), (65, 13)],                      # K > 64
])
@pytest.mark.parametrize("form", ["auto", "fp64"])
def test_batch_adjoint_matches_single_system(sizes, form):
    from juesgpu import MollerPlesset as mp, _lib
    sy = []
    for k, (n, o) in enumerate(sizes):
        s = make_system(n, o, 3 * n, seed=40 + k)
        sy.append((np.asfortranarray(s.ao_eri()), np.asfortranarray(s.C), o, s.eps))
    ctx = _lib.context(0)
    ctx.set_batch_form(form)
    try:
        e, gbs, cbs, info = mp.batch_rmp2(sy, adjoint=True, e_bar=0.5)
    finally:
        ctx.set_batch_form("auto")
    shapes = [info.tile_shape[k] for k in range(info.nstages)]
    assert info.nstages == 12 and shapes[11] < 4
    assert (max(shapes) < 4) if form == "fp64" else (shapes[0] == 5 and shapes[7] == 5)
    for (g, C, o, eps), eb, gb, cb in zip(sy, e, gbs, cbs):
        E, gs, cs = mp.rmp2_adjoint(gao=g, C=C, nocc=o, eps=eps, e_bar=0.5)
        assert abs(E - eb) < 1e-13 * max(1.0, abs(E))
        assert np.abs(gb - gs).max() < 1e-13 * np.abs(gs).max()
        assert np.abs(cb - cs).max() < 1e-13 * np.abs(cs).max()
