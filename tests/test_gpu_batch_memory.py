"""Device memory of the batched form: its stages run one after another and share one set of digit planes, and an idle
plan makes room for other calls."""
import numpy as np
import pytest

from test_gpu_pack_memory import MB, gemm, least_limit, mock
from juesgpu.synthetic import make_system

pytestmark = pytest.mark.gpu


def systems(count, n, o):
    out = []
    for k in range(count):
        s = make_system(n, o, 3 * n, seed=50 + k)
        out.append((np.asfortranarray(s.ao_eri()), np.asfortranarray(s.C), o, s.eps))
    return out


def batch(ctx, sy):
    """the stages' forms, or False where the memory limit refuses the call"""
    from juesgpu import MollerPlesset, _lib
    try:
        with mock.patch.object(_lib, "context", lambda device=0: ctx):
            info = MollerPlesset.batch_rmp2(sy, adjoint=True)[3]
    except _lib.JuESError as e:
        assert e.code == _lib.ENOMEM
        return False
    return [info.tile_shape[k] for k in range(info.nstages)]


def test_stages_share_their_planes():
    from juesgpu import _lib
    n, o, count = 40, 8, 6
    sy = systems(count, n, o)
    ctx = _lib.Context(0)
    try:
        digits = [k for k, f in enumerate(batch(ctx, sy)) if f == 5]
    finally:
        ctx.close()
    assert {0, 7, 8, 9} <= set(digits)

    def all_digits(ctx):
        forms = batch(ctx, sy)
        return bool(forms) and all(forms[k] == 5 for k in digits)

    plain, full = least_limit(lambda ctx: bool(batch(ctx, sy))), least_limit(all_digits)
    # 15 bytes an element of a stage's operands; the first third-quarter launch has the two largest, n^3 rows of n
    # and o n^2 rows of n (48 padded); exponents, lists, tables and smaller sides below 10 %
    largest = 15 * 48 * count * (n ** 3 + o * n ** 2)
    assert (full - plain) * MB <= 1.1 * largest + 4 * MB


def test_idle_plan_makes_room():
    from juesgpu import _lib
    rng = np.random.default_rng(1)
    A, B = np.asfortranarray(rng.normal(size=(20000, 500))), np.asfortranarray(rng.normal(size=(500, 300)))
    limit = least_limit(lambda ctx: gemm(ctx, A, B, 1))
    ctx = _lib.Context(0)
    try:
        sy = systems(6, 40, 8)
        first = batch(ctx, sy)
        ctx.set_mem_limit((limit + 1) * MB)
        assert gemm(ctx, A, B, 1)
        ctx.set_mem_limit(0)
        assert batch(ctx, sy) and first   # built again
    finally:
        ctx.close()
