"""Device memory of the digit planes: whatever a context ran before, a call that fits its memory limit in a fresh
context still fits, and an FP64 solve keeps the tensor-core form where its planes cannot all be kept.
"""
import ctypes as C
from unittest import mock

import numpy as np
import pytest

from juesgpu.synthetic import make_system

pytestmark = pytest.mark.gpu

MB = 1 << 20


def cc_solve(ctx, n, o, precision, sweeps=2):
    """energy and amplitudes of a CCD session that is closed again; False where the memory limit refuses it"""
    from juesgpu import _lib
    from juesgpu.CoupledCluster import CCSession
    sy = make_system(n, o, 3 * n, seed=9)
    try:
        with mock.patch.object(_lib, "context", lambda device=0: ctx):
            s = CCSession(0, gao=np.asfortranarray(sy.ao_eri()), Cocc=np.asfortranarray(sy.C[:, :o]),
                          Cvir=np.asfortranarray(sy.C[:, o:]), eps=sy.eps, maxit=sweeps, r_conv=0.0,
                          precision=precision, refine=0)
        try:
            s.iterate(sweeps)
            return s.energy(), s.amplitudes()[1]
        finally:
            s.close()
    except _lib.JuESError as e:
        assert e.code == _lib.ENOMEM
        return False


def gemm(ctx, A, B, precision):
    from juesgpu import _lib
    out = np.zeros((A.shape[0], B.shape[1]), order="F")
    st = ctx.lib.jues_gemm(ctx.h, 0, 0, A.shape[0], B.shape[1], A.shape[1], C.c_double(1.0), _lib.ptr(A), A.shape[0],
                           _lib.ptr(B), B.shape[0], C.c_double(0.0), _lib.ptr(out), A.shape[0], precision)
    assert st in (0, _lib.ENOMEM)
    return st == 0


def least_limit(call):
    """the smallest limit, in MB, under which call(ctx) runs in a fresh context"""
    from juesgpu import _lib
    lo, hi = 1, 4096
    while hi - lo > 1:
        mid = (lo + hi) // 2
        ctx = _lib.Context(0)
        try:
            ctx.set_mem_limit(mid * MB)
            ok = call(ctx)
        finally:
            ctx.close()
        lo, hi = (lo, mid) if ok else (mid, hi)
    return hi


def test_closed_fp64_solves_leave_no_planes_behind():
    from juesgpu import _lib

    def call(ctx):
        return bool(cc_solve(ctx, 40, 8, "split"))

    limit = least_limit(call)
    ctx = _lib.Context(0)
    try:
        for n, o in ((44, 9), (52, 10), (60, 12)):
            assert cc_solve(ctx, n, o, "fp64")
        ctx.set_mem_limit((limit + 1) * MB)
        assert call(ctx)
    finally:
        ctx.close()


def test_idle_fp64_planes_make_room_for_a_split_product():
    from juesgpu import _lib
    rng = np.random.default_rng(1)
    A, B = np.asfortranarray(rng.normal(size=(6000, 500))), np.asfortranarray(rng.normal(size=(500, 300)))
    limit = least_limit(lambda ctx: gemm(ctx, A, B, 1))
    ctx = _lib.Context(0)
    try:
        assert gemm(ctx, np.asfortranarray(A[:1000]), B, 0)   # 10 MB of planes: in the way of the packs, not of the operands
        ctx.set_mem_limit((limit + 1) * MB)
        assert gemm(ctx, A, B, 1)
    finally:
        ctx.close()


def test_planes_that_cannot_be_kept_are_formed_again():
    # the largest planes, of the AO integrals, take 80 MB: with 100 MB beyond what the solve cannot do without,
    # every contraction's planes fit by themselves, and the results are bit by bit those without a limit
    from juesgpu import _lib
    n, o = 48, 10
    limit = least_limit(lambda ctx: bool(cc_solve(ctx, n, o, "fp64")))
    free, tight = _lib.Context(0), _lib.Context(0)
    try:
        want = cc_solve(free, n, o, "fp64", sweeps=3)
        tight.set_mem_limit((limit + 100) * MB)
        got = cc_solve(tight, n, o, "fp64", sweeps=3)
        assert got[0] == want[0] and np.array_equal(got[1], want[1])
    finally:
        free.close()
        tight.close()


def test_folded_ladders_do_not_depend_on_planes_held_before():
    # the smallest limit after the set-up under which the first sweep still folds the ladders, told by the last
    # bits of the amplitudes; with 250 MB more of another product's planes than the set-up leaves it folds under the same limit
    from juesgpu import _lib
    from juesgpu.CoupledCluster import CCSession
    n, o = 78, 18
    sy = make_system(n, o, 3 * n, seed=3)
    g = np.asfortranarray(sy.ao_eri())
    rng = np.random.default_rng(2)
    A, B = np.asfortranarray(rng.normal(size=(130000, 400))), np.asfortranarray(rng.normal(size=(400, 32)))

    def sweep(limit, product=False):
        ctx = _lib.Context(0)
        try:
            with mock.patch.object(_lib, "context", lambda device=0: ctx):
                s = CCSession(0, gao=g, Cocc=np.asfortranarray(sy.C[:, :o]), Cvir=np.asfortranarray(sy.C[:, o:]),
                              eps=sy.eps, maxit=2, r_conv=0.0, precision="fp64")
            try:
                if product:
                    assert gemm(ctx, A, B, 0)
                ctx.set_mem_limit(limit * MB)
                s.iterate(1)
                ctx.set_mem_limit(0)
                return s.amplitudes()[1]
            except _lib.JuESError as e:
                assert e.code == _lib.ENOMEM
                return None
            finally:
                s.close()
        finally:
            ctx.close()

    want = sweep(0)
    lo, hi = 1, 8192
    while hi - lo > 8:
        mid = (lo + hi) // 2
        got = sweep(mid)
        lo, hi = (lo, mid) if got is not None and np.array_equal(got, want) else (mid, hi)
    got = sweep(hi - 16)
    assert got is None or not np.array_equal(got, want)   # below the line the bits do differ
    assert np.array_equal(sweep(hi + 8, product=True), want)
