"""The calls whose speed is followed, through the package's public entry points.

Systems come from the synthetic generator's distribution (AO integrals B^T B with B ~ N(0, 0.15/sqrt(naux)),
naux = 3 nbf, orthonormal orbitals, occupied energies in [-2, -0.5], virtual in [0.2, 3]), drawn on
the GPU from the seed alone.  Unless a case says otherwise the arrays are host (numpy) arrays, as
the drop-in entry points take them.
"""
import math
import os
import sys
import warnings

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jues.jl_gb300"))

from juesgpu import MollerPlesset, IntegralTransformation  # noqa: E402
from juesgpu.CoupledCluster import CCSession, PerturbativeTriples, RCCSD, mRCCD  # noqa: E402
from juesgpu.Wavefunction import wfn_from_rhf  # noqa: E402

F64 = torch.float64


# ------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest named system (nbf=25): a single-point MP2, where launches and copies are all
        {"name": "mp2_25", "kind": "mp2", "n": 25, "o": 5, "precision": "fp64"},
        # MP2 at the size of the FP64 drop-in configuration (nbf=100)
        {"name": "mp2_100", "kind": "mp2", "n": 100, "o": 20, "precision": "fp64"},
        # an integral block for a user's own code: the largest block, ragged extents
        {"name": "eri_vvvv_77", "kind": "eri", "n": 77, "o": 15, "spec": "VVVV", "precision": "fp64"},
        # the backward path of MP2 at the differentiation configuration (nbf=120)
        {"name": "mp2_grad_120", "kind": "grad", "n": 120, "o": 25, "precision": "fp64"},
        # many small systems of uneven size, energies and gradients in one call
        {"name": "mp2_batch_24", "kind": "batch", "count": 24, "nmin": 10, "nmax": 60, "sizes": 1,
         "precision": "fp64"},
        # a small CCD solve: twelve sweeps of small kernels, bound by launches and synchronisations
        {"name": "ccd_25", "kind": "ccd", "n": 25, "o": 5, "sweeps": 12, "precision": "fp64", "refine": 0},
        # the FP64 drop-in configuration of CCD (nbf=100, DIIS)
        {"name": "ccd_100", "kind": "ccd", "n": 100, "o": 20, "sweeps": 8, "precision": "fp64", "refine": 0},
        # the split form as the mirror runs it by default: split sweeps, then two closing FP64 sweeps
        {"name": "ccd_90_split", "kind": "ccd", "n": 90, "o": 17, "sweeps": 40, "precision": "split", "refine": 2},
        # the precision configuration (nbf=200) from AO integrals already on the GPU
        {"name": "ccd_200_split", "kind": "ccd_dev", "n": 200, "o": 40, "sweeps": 10, "precision": "split"},
        # CCSD as the reference runs it (no DIIS), odd extents
        {"name": "ccsd_63", "kind": "ccsd", "n": 63, "o": 13, "sweeps": 6, "precision": "fp64"},
        # CCSD in the split form
        {"name": "ccsd_120_split", "kind": "ccsd", "n": 120, "o": 24, "sweeps": 6, "precision": "split"},
        # the (T) correction from host amplitudes and integrals
        {"name": "pt_12_48", "kind": "pt", "o": 12, "v": 48, "precision": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mp2", "eri", "grad", "batch", "ccd", "ccd_split", "ccd_dev", "ccsd", "ccsd_split", "pt"])

    def size(lo, hi):
        n = _log_int(rng, lo, hi)
        return {"n": n, "o": max(2, int(round(n * rng.uniform(0.12, 0.28))))}

    if kind == "mp2":
        return {"kind": "mp2", **size(14, 110), "precision": rng.choice(["fp64", "fp64", "split"])}
    if kind == "eri":
        spec = rng.choice(["OOVV", "OVOV", "OVVO", "OOOV", "OVVV", "VVVV"])
        return {"kind": "eri", **size(14, 90), "spec": spec, "precision": rng.choice(["fp64", "fp64", "split"])}
    if kind == "grad":
        return {"kind": "grad", **size(14, 115), "precision": rng.choice(["fp64", "fp64", "split"])}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 24), "nmin": 10, "nmax": rng.randint(16, 60),
                "sizes": rng.randint(0, 10 ** 6), "precision": "fp64"}
    if kind == "ccd":
        return {"kind": "ccd", **size(14, 96), "sweeps": rng.randint(3, 8), "precision": "fp64", "refine": 0}
    if kind == "ccd_split":
        return {"kind": "ccd", **size(40, 96), "sweeps": 40, "precision": "split", "refine": rng.choice([0, 2])}
    if kind == "ccd_dev":
        return {"kind": "ccd_dev", **size(60, 190), "sweeps": rng.randint(4, 10), "precision": "split"}
    if kind == "ccsd":
        return {"kind": "ccsd", **size(14, 63), "sweeps": rng.randint(3, 6), "precision": "fp64"}
    if kind == "ccsd_split":
        return {"kind": "ccsd", **size(48, 120), "sweeps": rng.randint(3, 6), "precision": "split"}
    return {"kind": "pt", "o": rng.randint(3, 12), "v": _log_int(rng, 12, 48),
            "precision": rng.choice(["fp64", "fp64", "split"])}


# ---------------------------------------------------------------------------------------- inputs
def _system(n, o, seed):
    """AO integrals (n^4 on the GPU, column-major meaning), orbitals C (n x n) and energies."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * n + 1009 * o + int(seed))
    naux = 3 * n
    x = torch.randn(naux, n, n, dtype=F64, device="cuda", generator=gen) * (0.15 / math.sqrt(naux))
    b = torch.triu(x)
    b = (b + torch.triu(x, 1).transpose(1, 2)).reshape(naux, n * n)
    g = b.T @ b
    c, _ = torch.linalg.qr(torch.randn(n, n, dtype=F64, device="cuda", generator=gen))
    eo = torch.sort(torch.rand(o, dtype=F64, device="cuda", generator=gen) * 1.5 - 2.0).values
    ev = torch.sort(torch.rand(n - o, dtype=F64, device="cuda", generator=gen) * 2.8 + 0.2).values
    return g, c, torch.cat([eo, ev])


def _host_wfn(n, o, seed):
    g, c, eps = _system(n, o, seed)
    # a symmetric n^2 x n^2 matrix: its transpose read column-major is the n^4 array
    gh = g.cpu().numpy().T.reshape(n, n, n, n, order="F")
    return wfn_from_rhf(c.cpu().numpy(), eps.cpu().numpy(), gh, o)


def _batch_sizes(case):
    r = np.random.default_rng(case["sizes"])
    ns = [int(x) for x in r.integers(case["nmin"], case["nmax"] + 1, size=case["count"])]
    return [(n, max(1, int(round(n / 5)))) for n in ns]


def _pt_inputs(o, v, seed):
    """Amplitudes and integrals of the magnitudes a CCSD on the generator's systems meets."""
    gen = torch.Generator(device="cuda").manual_seed(7919 * o + 104729 * v + int(seed))

    def rnd(*shape, scale=1.0):
        return torch.randn(*shape, dtype=F64, device="cuda", generator=gen) * scale

    t1 = rnd(o, v, scale=2e-3)
    x = rnd(o, o, v, v, scale=4e-3)
    t2 = x + x.permute(1, 0, 3, 2)
    naux = 3 * (o + v)
    s = 0.15 / math.sqrt(naux)
    bvv, bvo, boo = rnd(naux, v, v, scale=s), rnd(naux, v, o, scale=s), rnd(naux, o, o, scale=s)
    bvv, boo = (bvv + bvv.transpose(1, 2)) / 2 ** 0.5, (boo + boo.transpose(1, 2)) / 2 ** 0.5
    vvvo = torch.einsum("Pab,Pci->abci", bvv, bvo)
    vooo = torch.einsum("Pai,Pjk->aijk", bvo, boo)
    vovo = torch.einsum("Pai,Pbj->aibj", bvo, bvo)
    fo = torch.sort(torch.rand(o, dtype=F64, device="cuda", generator=gen) * 1.5 - 2.0).values
    fv = torch.sort(torch.rand(v, dtype=F64, device="cuda", generator=gen) * 2.8 + 0.2).values
    return {"T1": t1, "T2": t2, "Vvvvo": vvvo, "Vvooo": vooo, "Vvovo": vovo, "fo": fo, "fv": fv}


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("mp2", "eri", "grad", "ccd", "ccsd"):
        st["wfn"] = _host_wfn(case["n"], case["o"], seed)
    elif kind == "batch":
        st["systems"] = [_host_wfn(n, o, 1000 * seed + k) for k, (n, o) in enumerate(_batch_sizes(case))]
    elif kind == "ccd_dev":
        g, c, eps = _system(case["n"], case["o"], seed)
        st["g"] = g
        c = c.cpu().numpy()
        st["Cocc"] = np.asfortranarray(c[:, :case["o"]])
        st["Cvir"] = np.asfortranarray(c[:, case["o"]:])
        st["eps"] = eps.cpu().numpy()
        torch.cuda.synchronize()   # the library reads g on its own stream
    else:
        st["args"] = {k: np.asfortranarray(t.cpu().numpy()) for k, t in
                      _pt_inputs(case["o"], case["v"], seed).items()}
    return st


# ------------------------------------------------------------------------------------- the calls
def run(state):
    case = state["case"]
    kind, prec = case["kind"], case["precision"]
    if kind == "mp2":
        return MollerPlesset.do_rmp2(state["wfn"], precision=prec)
    if kind == "eri":
        return IntegralTransformation.get_eri(state["wfn"], case["spec"], precision=prec)
    if kind == "grad":
        return MollerPlesset.rmp2_adjoint(state["wfn"], precision=prec)
    if kind == "batch":
        e, gb, cb, _ = MollerPlesset.batch_rmp2(state["systems"], adjoint=True, precision=prec)
        return e, gb, cb
    if kind == "ccd":
        if prec == "fp64":
            return mRCCD.do_rccd(state["wfn"], maxit=case["sweeps"], r_conv=0.0, return_T2=True)
        return mRCCD.do_rccd(state["wfn"], maxit=case["sweeps"], precision=prec, refine=case["refine"],
                             r_conv=1e-6, return_T2=True)
    if kind == "ccd_dev":
        s = CCSession(0, gao_dev_ptr=state["g"].data_ptr(), Cocc=state["Cocc"], Cvir=state["Cvir"], eps=state["eps"],
                      maxit=case["sweeps"], r_conv=0.0, precision=prec, refine=0)
        s.iterate(case["sweeps"])
        e, t2 = s.energy(), s.amplitudes()[1]
        s.close()
        return e, t2
    if kind == "ccsd":
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")   # a fixed number of sweeps
            return RCCSD.do_rccsd(state["wfn"], maxit=case["sweeps"], precision=prec, return_T1=True)
    return PerturbativeTriples.compute_pT(**state["args"], precision=prec)


# -------------------------------------------------------------------------------- least work done
def _transform_flops(n, d):
    f, prod, left = 0.0, 1.0, float(n) ** 4
    for x in sorted(d):
        prod *= x
        left /= n
        f += 2.0 * left * n * prod
    return f


def _dims(spec, o, v):
    return [o if ch in "oO" else v for ch in spec]


def _ccd_flops(o, v):
    """One sweep: both ladders over pairs of equal symmetry, six ring contractions, X."""
    return 0.5 * o * o * v ** 4 + 12.0 * o ** 3 * v ** 3 + 1.5 * o ** 4 * v * v


def work(case):
    kind = case["kind"]
    if kind == "pt":
        o, v = case["o"], case["v"]
        words = o * v + (o * v) ** 2 * 2 + v ** 3 * o + v * o ** 3 + o + v
        return {"bytes": 8.0 * words, "flops": 2.0 * o * (o + 1) * (o + 2) * v ** 3 * (v + o)}
    if kind == "batch":
        b = f = 0.0
        for n, o in _batch_sizes(case):
            w = work({"kind": "grad", "n": n, "o": o})
            b, f = b + w["bytes"], f + w["flops"]
        return {"bytes": b, "flops": f}
    n, o = case["n"], case["o"]
    v, n4 = n - o, float(n) ** 4
    if kind == "mp2":
        return {"bytes": 8.0 * (n4 + n * n + n), "flops": _transform_flops(n, (o, o, v, v))}
    if kind == "eri":
        d = _dims(case["spec"], o, v)
        return {"bytes": 8.0 * (n4 + n * n + float(np.prod(d))), "flops": _transform_flops(n, d)}
    if kind == "grad":
        f = 2 * _transform_flops(n, (o, o, v, v)) + 2.0 * o * o * v * n * n * (v + n)
        return {"bytes": 8.0 * (2 * n4 + 2 * n * n + n), "flops": f}
    blocks = ["OOVV", "OVOV", "OOOO", "VVVV"] + (["OOOV", "OVVV"] if kind == "ccsd" else ["OVVO"])
    # the blocks share quarter steps; the largest alone is what cannot be left out
    f = _transform_flops(n, _dims("VVVV", o, v))
    sweeps = case["sweeps"] if case["sweeps"] < 40 else 8   # a converged solve takes about eight
    per = _ccd_flops(o, v) + (o * o * v ** 3 * o * 1.0 if kind == "ccsd" else 0.0)
    once = sum(float(np.prod(_dims(b, o, v))) for b in blocks)
    return {"bytes": 8.0 * (n4 + n * n + n + 2.0 * (o * v) ** 2 + sweeps * once), "flops": f + sweeps * per}


# ------------------------------------------------------------------- the same in plain 64-bit torch
def _mo(g4, *cs):
    """(pq|rs) of the AO integrals g4[m,n,l,s], one index after the other."""
    x = g4
    for c in cs:
        x = torch.tensordot(x, c, dims=([0], [0]))   # contracts the first index, appends the new one
    return x


def _exact_system(n, o, seed):
    g, c, eps = _system(n, o, seed)
    return g.reshape(n, n, n, n), c, eps


def _ediff(eps, o):
    eo, ev = eps[:o], eps[o:]
    return (eo[:, None, None, None] + eo[None, :, None, None] - ev[None, None, :, None]
            - ev[None, None, None, :])


def _mp2(g4, c, eps, o):
    k = _mo(g4, c[:, :o], c[:, o:], c[:, :o], c[:, o:]).permute(0, 2, 1, 3)   # <ij|ab>
    return (k * (2 * k - k.transpose(2, 3)) / _ediff(eps, o)).sum()


def _mp2_grad(n, o, seed):
    g4, c, eps = _exact_system(n, o, seed)
    with torch.enable_grad():
        g4.requires_grad_(True)
        c.requires_grad_(True)
        e = _mp2(g4, c, eps, o)
        gg, gc = torch.autograd.grad(e, (g4, c))
    return float(e.detach()), gg.cpu().numpy(), gc.cpu().numpy()


def _phys(g4, c, o, spec):
    cs = [c[:, :o] if ch in "oO" else c[:, o:] for ch in spec]
    return _mo(g4, cs[0], cs[2], cs[1], cs[3]).permute(0, 2, 1, 3).contiguous()


class _Diis:
    """Up to five (amplitude, error) pairs, the error's Gram matrix scaled by its largest entry."""

    def __init__(self):
        self.v, self.e = [], []

    def step(self, new, old):
        self.v.append(new)
        self.e.append(new - old)
        self.v, self.e = self.v[-5:], self.e[-5:]
        m = len(self.v)
        b = np.full((m + 1, m + 1), -1.0)
        b[m, m] = 0.0
        for i in range(m):
            for j in range(m):
                b[i, j] = float(torch.dot(self.e[i], self.e[j]))
        b[:m, :m] /= np.abs(b[:m, :m]).max()
        rhs = np.zeros(m + 1)
        rhs[m] = -1.0
        w = np.linalg.solve(b, rhs)
        return sum(float(w[i]) * self.v[i] for i in range(m)), float(self.e[-1].norm())


def _ccd_sweep(t, oovv, ovov, ovvo, oooo, vvvv, d):
    es = torch.einsum
    tt = 2 * t - t.transpose(0, 1)
    fae = -es("mnef,mnaf->ae", oovv, tt)
    fmi = es("mnef,inef->mi", oovv, 2 * t - t.transpose(2, 3))
    x = oooo + es("mnef,ijef->mnij", oovv, t)
    wj = ovvo + 0.5 * es("mnef,njfb->mbej", oovv, tt) - 0.5 * es("nmef,njfb->mbej", oovv, t)
    wk = -ovov.transpose(2, 3) + 0.5 * es("jnfb,nmef->mbej", t, oovv)
    z = (es("ijae,be->ijab", t, fae) - es("imab,mj->ijab", t, fmi) + es("imae,mbej->ijab", t, 2 * wj + wk)
         - es("miae,mbej->ijab", t, wj) + es("mibe,maej->ijab", t, wk))
    r = oovv + es("mnij,mnab->ijab", x, t) + es("ijef,abef->ijab", t, vvvv) + z + z.permute(1, 0, 3, 2)
    return r / d


def _ccd(case, seed):
    n, o = case["n"], case["o"]
    g4, c, eps = _exact_system(n, o, seed)
    oovv, ovov, ovvo, oooo, vvvv = (_phys(g4, c, o, s) for s in ("OOVV", "OVOV", "OVVO", "OOOO", "VVVV"))
    del g4
    d = _ediff(eps, o)
    t = torch.zeros_like(oovv)
    diis = _Diis()
    last = 0.0 if case["precision"] == "fp64" or case["kind"] == "ccd_dev" else 1e-12   # the split solve ends converged
    for _ in range(case["sweeps"]):
        x, step = diis.step(_ccd_sweep(t, oovv, ovov, ovvo, oooo, vvvv, d).reshape(-1), t.reshape(-1))
        t = x.reshape(t.shape)
        if step < last:
            break
    return float((oovv * (2 * t - t.transpose(0, 1))).sum()), t.cpu().numpy()


def _ccsd(case, seed):
    n, o = case["n"], case["o"]
    g4, c, eps = _exact_system(n, o, seed)
    oooo, ooov, oovv, ovov, ovvv, vvvv = (_phys(g4, c, o, s) for s in ("OOOO", "OOOV", "OOVV", "OVOV", "OVVV", "VVVV"))
    del g4
    es = torch.einsum
    d, dia = _ediff(eps, o), eps[:o, None] - eps[None, o:]
    w2 = 2 * oovv - oovv.transpose(0, 1)
    t2 = oovv / d
    t1 = torch.zeros(o, n - o, dtype=F64, device="cuda")
    for _ in range(case["sweeps"]):
        tt = es("ia,jb->ijab", t1, t1)
        ta, th = t2 + tt, t2 + 0.5 * tt
        fae = es("mf,mafe->ae", t1, 2 * ovvv) - es("mf,maef->ae", t1, ovvv) - es("mnaf,mnef->ae", th, w2)
        fmi = (es("ne,mnie->mi", t1, 2 * ooov) - es("ne,nmie->mi", t1, ooov)
               + es("inef,mnef->mi", th, 2 * oovv - oovv.transpose(2, 3)))
        fme = es("nf,mnef->me", t1, w2)
        wm = (oooo + es("je,mnie->mnij", t1, ooov) + es("ie,nmje->mnij", t1, ooov)
              + es("ijef,mnef->mnij", ta, oovv))   # the ladder term of Wabef's T part included
        y = es("ijef,mafe->ijam", ta, ovvv)
        wj = (oovv.permute(0, 3, 2, 1) + es("jf,mbef->mbej", t1, ovvv) - es("nb,nmje->mbej", t1, ooov)
              - 0.5 * es("jnfb,mnef->mbej", t2 + 2 * tt, oovv) + 0.5 * es("njfb,mnef->mbej", t2, w2))
        wk = (-ovov.transpose(2, 3) - es("jf,mbfe->mbej", t1, ovvv) + es("nb,mnje->mbej", t1, ooov)
              + es("jnfb,nmef->mbej", 0.5 * t2 + tt, oovv))
        r1 = (es("ie,ae->ia", t1, fae) - es("ma,mi->ia", t1, fmi) + es("me,imae->ia", fme, 2 * t2 - t2.transpose(0, 1))
              + es("me,imae->ia", t1, 2 * oovv) - es("me,maie->ia", t1, ovov)
              - es("mnae,mnie->ia", t2, 2 * ooov - ooov.transpose(0, 1))
              + es("imef,mafe->ia", t2, 2 * ovvv) - es("imef,maef->ia", t2, ovvv))
        z = (es("ijae,be->ijab", t2, fae - 0.5 * es("mb,me->be", t1, fme))
             - es("imab,mj->ijab", t2, fmi + 0.5 * es("je,me->mj", t1, fme))
             - es("ijam,mb->ijab", y, t1)
             + es("imae,mbej->ijab", t2, 2 * wj + wk) - es("miae,mbej->ijab", t2, wj)
             + es("mibe,maej->ijab", t2, wk)
             - es("imea,mjeb->ijab", tt, oovv) - es("imeb,maje->ijab", tt, ovov)
             + es("ie,jabe->ijab", t1, ovvv) - es("ma,mjib->ijab", t1, ooov))
        r2 = oovv + es("mnab,mnij->ijab", ta, wm) + es("ijef,abef->ijab", ta, vvvv) + z + z.permute(1, 0, 3, 2)
        t1, t2 = r1 / dia, r2 / d
    x = t2 + es("ia,jb->ijab", t1, t1)
    return float((oovv * (2 * x - x.transpose(0, 1))).sum()), t1.cpu().numpy(), t2.cpu().numpy()


def _pt(case, seed):
    a = _pt_inputs(case["o"], case["v"], seed)
    t1, t2, vv, vo, ov = a["T1"], a["T2"], a["Vvvvo"], a["Vvooo"], a["Vvovo"]
    fo, fv = a["fo"], a["fv"]
    o, v = t1.shape
    es = torch.einsum
    ar = torch.arange(v, device="cuda")
    keep = (ar[:, None, None] >= ar[None, :, None]) & (ar[None, :, None] >= ar[None, None, :])
    same = (1.0 + (ar[:, None, None] == ar[None, :, None]).to(F64) + (ar[None, :, None] == ar[None, None, :]).to(F64))
    dv = fv[:, None, None] + fv[None, :, None] + fv[None, None, :]
    total = 0.0
    for i in range(o):
        for j in range(i + 1):
            for k in range(j + 1):
                w = 0.0
                # (p,q,r) runs over the orderings of (i,a), (j,b), (k,c)
                lab = {i_: x for i_, x in zip((0, 1, 2), "abc")}
                occ = (i, j, k)
                for p, q, r in ((0, 1, 2), (0, 2, 1), (2, 0, 1), (2, 1, 0), (1, 2, 0), (1, 0, 2)):
                    x, y, u = lab[p], lab[q], lab[r]
                    w = w + es(f"{y}d{x},{u}d->abc", vv[:, :, :, occ[p]], t2[occ[r], occ[q]])
                    w = w - es(f"{u}l,l{x}{y}->abc", vo[:, occ[r], occ[q], :], t2[occ[p]])
                z = (w + es("bc,a->abc", ov[:, j, :, k], t1[i]) + es("ac,b->abc", ov[:, i, :, k], t1[j])
                     + es("ab,c->abc", ov[:, i, :, j], t1[k]))

                def perm(t, s):
                    # element t[s of (a,b,c)] at [a,b,c]
                    return t.permute(*["abc".index(ch) for ch in s]) if s != "abc" else t
                inv = {"abc": "abc", "acb": "acb", "bac": "bac", "bca": "cab", "cab": "bca", "cba": "cba"}
                ws = {s: perm(w, inv[s]) for s in inv}
                zs = {s: perm(z, inv[s]) for s in inv}
                xx = sum(ws[s] * zs[s] for s in inv)
                yy, zz = zs["abc"] + zs["bca"] + zs["cab"], zs["acb"] + zs["bac"] + zs["cba"]
                en = ((yy - 2 * zz) * (ws["abc"] + ws["bca"] + ws["cab"])
                      + (zz - 2 * yy) * (ws["acb"] + ws["bac"] + ws["cba"]) + 3 * xx)
                den = (fo[i] + fo[j] + fo[k] - dv) * same
                total += float((en / den)[keep].sum()) * (2 - (i == j) - (j == k))
    return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "mp2":
        g4, c, eps = _exact_system(case["n"], case["o"], seed)
        return float(_mp2(g4, c, eps, case["o"]))
    if kind == "eri":
        g4, c, _ = _exact_system(case["n"], case["o"], seed)
        return _phys(g4, c, case["o"], case["spec"]).cpu().numpy()
    if kind == "grad":
        return _mp2_grad(case["n"], case["o"], seed)
    if kind == "batch":
        es, gbs, cbs = [], [], []
        for k, (n, o) in enumerate(_batch_sizes(case)):
            e, gb, cb = _mp2_grad(n, o, 1000 * seed + k)
            es.append(e)
            gbs.append(gb)
            cbs.append(cb)
        return np.array(es), gbs, cbs
    if kind in ("ccd", "ccd_dev"):
        return None if case["n"] > 130 else _ccd(case, seed)
    if kind == "ccsd":
        return _ccsd(case, seed)
    return _pt(case, seed)
