"""The batched form's choice between digit planes and FP64 tiles, by time on the data at hand: three systems of nbf 64
with 32 occupied, whose large stages are five times faster on the tensor cores, and the same systems in a graded basis
(integrals falling over 30 binades along each index, orbitals rising), where the digit form hands every tile back to
the FP64 pipe and takes a fifth longer than the FP64 tiles alone."""
import numpy as np
import pytest

from juesgpu.synthetic import make_system

pytestmark = pytest.mark.gpu


def system(seed, span, n=64, o=32):
    s = make_system(n, o, 3 * n, seed=seed)
    d = 2.0 ** np.rint(np.linspace(0, -span, n)[np.random.default_rng(seed).permutation(n)])
    g = s.ao_eri() * d[:, None, None, None] * d[None, :, None, None] * d[None, None, :, None] * d[None, None, None, :]
    return np.asfortranarray(g), np.asfortranarray(s.C / d[:, None]), o, s.eps


def test_digit_stages_are_chosen_by_time():
    from juesgpu import MollerPlesset as mp
    energies = {}
    for span, digits in ((0, True), (30, False)):
        from juesgpu import _lib
        ctx = _lib.context(0)
        for form in ("fp64", "auto"):
            ctx.set_batch_form(form)   # a plan of its own, tuned on these systems
            try:
                e, _, _, info = mp.batch_rmp2([system(k, span) for k in range(3)], adjoint=False)
            finally:
                ctx.set_batch_form("auto")
            energies[span, form] = e
        assert (info.tile_shape[0] == 5) == digits
        assert np.all(np.abs(energies[span, "auto"] - energies[span, "fp64"]) <= 1e-12 * np.abs(e))
    assert np.all(np.abs(energies[30, "fp64"] - energies[0, "fp64"]) <= 1e-12 * np.abs(energies[0, "fp64"]))
