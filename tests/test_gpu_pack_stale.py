"""Packs of a caller's device array do not outlive the call that formed them, also when it fails: a solve refused by
the memory limit after its integral transform, the array rewritten in place, and the solve repeated without the limit."""
import numpy as np
import pytest

from test_gpu_pack_memory import MB, mock
from juesgpu.synthetic import make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_rewritten_integrals_after_a_refused_solve(precision):
    torch = pytest.importorskip("torch")
    from juesgpu import _lib
    from juesgpu.CoupledCluster import CCSession
    n, o = 40, 8
    one, two = make_system(n, o, 3 * n, seed=1), make_system(n, o, 3 * n, seed=2)
    gao = [torch.from_numpy(np.ascontiguousarray(s.ao_eri().T)).cuda() for s in (one, two)]
    buf = torch.empty_like(gao[0])

    def energy(ctx, sy):
        with mock.patch.object(_lib, "context", lambda device=0: ctx):
            s = CCSession(0, gao_dev_ptr=buf.data_ptr(), Cocc=np.asfortranarray(sy.C[:, :o]),
                          Cvir=np.asfortranarray(sy.C[:, o:]), eps=sy.eps, maxit=2, r_conv=0.0, precision=precision,
                          refine=0)
        try:
            s.iterate(2)
            return s.energy()
        finally:
            s.close()

    def run(limits, arrays):
        ctx = _lib.Context(0)
        e = None
        try:
            for limit, k in zip(limits, arrays):
                buf.copy_(gao[k])
                torch.cuda.synchronize()
                ctx.set_mem_limit(limit * MB)
                try:
                    e = energy(ctx, (one, two)[0])   # the same orbitals: only the array's values differ
                except _lib.JuESError as err:
                    assert err.code == _lib.ENOMEM
                    e = None
            return e
        finally:
            ctx.close()

    least = next(m for m in range(1, 400) if run([m], [0]) is not None)
    want = run([0], [1])
    refused = 0
    for m in range(least - 1, max(0, least - 40), -2):   # refused at later and earlier points of the set-up
        assert run([m, 0], [0, 1]) == want
        refused += 1
    assert refused > 2
