"""(T) with amplitudes of any size beside the integrals: the stacked contractions scale them to the integrals' size by
a power of two, so amplitudes 2^-k times as large give exactly 2^-2k times the energy (without T1 the energy is
quadratic in T2).  Where digits of the smaller half were cut off, or the contractions redone on the FP64 pipe, the
last bits differ.  The split form is held to 2^-18 of the FP64 energy: its elements keep K 2^-18 of their magnitudes at
worst, and independent roundings average over them.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def inputs(o, v, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(o, o, v, v)) * 4e-3
    z = rng.normal(size=(v, v, v, o)) * 2e-3
    y = rng.normal(size=(v, o, v, o)) * 2e-3
    kw = dict(T1=np.zeros((o, v)), T2=x + x.transpose(1, 0, 3, 2), Vvvvo=z + z.transpose(1, 0, 2, 3),
              Vvooo=2e-3 * rng.normal(size=(v, o, o, o)), Vvovo=y + y.transpose(2, 3, 0, 1), fo=-1.0 - rng.random(o),
              fv=0.5 + rng.random(v))
    return {k: np.asfortranarray(a) for k, a in kw.items()}


@pytest.mark.parametrize("o,v", [(3, 17), (7, 40)])
def test_pT_amplitudes_of_any_size(o, v):
    from juesgpu.CoupledCluster import PerturbativeTriples
    kw = inputs(o, v, 3)
    base = {p: PerturbativeTriples.compute_pT(precision=p, **kw) for p in ("fp64", "split")}
    assert abs(base["split"] - base["fp64"]) <= 2.0 ** -18 * abs(base["fp64"])
    t2 = kw.pop("T2")
    for k in (-6, 4, 7, 9, 12, 24, 50):
        for p, e in base.items():
            got = PerturbativeTriples.compute_pT(precision=p, T2=np.asfortranarray(t2 * 2.0 ** -k), **kw)
            assert got * 2.0 ** (2 * k) == e


def test_pT_without_amplitudes_or_integrals():
    from juesgpu.CoupledCluster import PerturbativeTriples
    for name in ("T2", "Vvvvo", "Vvooo"):
        kw = inputs(3, 12, 4)
        kw[name] = np.zeros_like(kw[name])
        e = {p: PerturbativeTriples.compute_pT(precision=p, **kw) for p in ("fp64", "split")}
        assert np.isfinite(e["fp64"]) and abs(e["split"] - e["fp64"]) <= 2.0 ** -18 * abs(e["fp64"])


@pytest.mark.parametrize("every", [2, 5, 16])
def test_pT_graded_amplitudes(every):
    # amplitudes and integrals of some virtual orbitals 2^-14 and 2^-30 times the others': the grouped contractions leave
    # out single elements and whole half tiles; bounds as at the edges (1e-11 FP64, 1e-6 split)
    from juesgpu.CoupledCluster import PerturbativeTriples
    from oracle import triples
    o, v = 4, 37
    kw = inputs(o, v, every)
    d = np.where(np.arange(v) % every == 0, 2.0 ** -14, 1.0)
    f = np.where(np.arange(v) % every == 1, 2.0 ** -30, 1.0)
    kw["T1"] = np.asfortranarray(np.random.default_rng(1).normal(size=(o, v)) * 1e-2)
    kw["T2"] = np.asfortranarray(kw["T2"] * d[:, None] * d)
    kw["Vvvvo"] = np.asfortranarray(kw["Vvvvo"] * f[:, None, None, None] * f[:, None, None])
    want = triples.compute_pT(**kw)
    assert abs(PerturbativeTriples.compute_pT(**kw) - want) <= 1e-11 * abs(want)
    assert abs(PerturbativeTriples.compute_pT(precision="split", **kw) - want) <= 1e-6 * abs(want)
