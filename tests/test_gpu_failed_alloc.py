"""A table build that runs out of device memory: the call returns PCG_ENOMEM, and
the calls after it on the same context build what they need and are right.
One allocation after another is refused, and a table is asked for that no GPU
holds."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

PCG_ERANGE, PCG_ENOMEM = 2, 3


def _noalloc(pcg, ctx, x):
    p, out = pcg.gourdon_params(x), pcg.I128()
    st = pcg.load().pcg_D_noalloc(ctx._h, pcg.to_i128(x), ctypes.c_int64(p["y"]), ctypes.c_int64(p["z"]),
                                  ctypes.c_int64(p["k"]), None, ctypes.byref(out))
    return st, pcg.from_i128(out)


def _small_calls(pcg, ctx, golden):
    """Calls that the tables of a context made for 1e12 serve: first what reads
    tables without building any, then the rest."""
    x = 10 ** 12
    st, v = _noalloc(pcg, ctx, x)
    assert st == PCG_ERANGE or (st == 0 and v == WANT["D"])
    assert pcg.D_default(x, ctx=ctx) == WANT["D"]
    assert pcg.pi(x, ctx=ctx) == golden["pi_pow10"][str(x)]
    assert pcg.phi(10 ** 10, 20, ctx=ctx) == WANT["phi"]
    assert pcg.pi_deleglise_rivat(10 ** 11, ctx=ctx) == golden["pi_pow10"][str(10 ** 11)]
    assert pcg.pi(5 * 10 ** 9, ctx=ctx) == 234954223
    for t in ("primes", "pi", "factor_d", "factor_dr"):
        ctx.read_table(t)


WANT = {}


@pytest.fixture(autouse=True)
def _want(pcg, ora):
    if not WANT:
        p = pcg.gourdon_params(10 ** 12)
        ctx = pcg.Context(0)
        WANT["D"] = ora.D(10 ** 12, p["y"], p["z"], p["k"], threads=8)[0]
        WANT["phi"] = pcg.phi(10 ** 10, 20, ctx=ctx)
        ctx.close()


def test_table_larger_than_any_gpu(pcg, golden):
    ctx = pcg.Context(10 ** 12)
    try:
        _small_calls(pcg, ctx, golden)
        for z in (10 ** 13, 3 * 10 ** 13):
            with pytest.raises(pcg.PrimecountError) as e:
                pcg.D(10 ** 20, 10 ** 6, z, 8, ctx=ctx)          # 8e12 bytes of FactorTable
            assert e.value.status == PCG_ENOMEM
            _small_calls(pcg, ctx, golden)
    finally:
        ctx.close()


BIG = {
    "pi": lambda p, c: p.pi(10 ** 16 + 10 ** 13, ctx=c),
    "pi_wide": lambda p, c: p.pi(10 ** 17, ctx=c),
    "dr": lambda p, c: p.pi_deleglise_rivat(10 ** 15, ctx=c),
    "phi_leaves": lambda p, c: p.phi(10 ** 15, 300, ctx=c),
    "phi_p2_p3": lambda p, c: p.phi(10 ** 14, 4000, ctx=c),
    "D": lambda p, c: p.D(10 ** 16, 2 * 10 ** 6, 4 * 10 ** 6, 8, ctx=c),
    "S2_hard": lambda p, c: p.S2_hard_default(10 ** 15, ctx=c),
}


@pytest.mark.parametrize("name", sorted(BIG))
def test_one_allocation_refused(pcg, golden, name):
    refuse = pcg.load().pcg_test_refuse_alloc
    refuse.argtypes, refuse.restype = [ctypes.c_int64], None
    fresh = pcg.Context(0)
    want = BIG[name](pcg, fresh)
    fresh.close()
    for n in range(1, 200):
        ctx = pcg.Context(10 ** 12)
        try:
            _small_calls(pcg, ctx, golden)
            refuse(n)
            try:
                got = BIG[name](pcg, ctx)
            except pcg.PrimecountError as e:
                assert e.status == PCG_ENOMEM, (n, e)
                got = None
            finally:
                refuse(0)
            if got is not None:                  # the call makes fewer than n allocations
                assert got == want
                break
            _small_calls(pcg, ctx, golden)
            assert BIG[name](pcg, ctx) == want, n
        finally:
            ctx.close()
    assert 3 < n < 199
