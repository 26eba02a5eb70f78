"""A context's memory budget and the FactorTable that pi(x) reads: from 3e16 on
z = 2 y while that table fits the budget, else z = y, and a call keeps what the
context was made with."""
import pytest

pytestmark = pytest.mark.gpu

X = 10 ** 17


def _sizes(pcg):
    """Device bytes of a context for X with the table of z = 2 y and of z = y."""
    ctx = pcg.Context(X)
    n, eb, lim = ctx.table_info("factor_d")
    wide = ctx.device_bytes()
    ctx.close()
    y = pcg.gourdon_params(X)["y"]
    assert (eb, lim) == (2, 2 * y)
    one = pcg.Context(0)
    pcg.D(X, y, y, 8, ctx=one)
    narrow = wide - 2 * (n - one.table_info("factor_d")[0])
    one.close()
    return y, wide, narrow


def test_budget_below_the_wide_table(pcg, golden):
    y, wide, narrow = _sizes(pcg)
    for budget in (wide - 1, (wide + narrow) // 2, narrow):
        ctx = pcg.Context(X, budget)
        try:
            assert ctx.table_info("factor_d")[2] == y
            for x in (X, X - 10 ** 16, X):
                p = pcg.pi(x, ctx=ctx)
                if x == X:
                    assert p == golden["pi_pow10"][str(X)]
                assert ctx.table_info("factor_d")[2] == y, budget      # no wider table built in the call
            assert pcg.pi(X, ctx=ctx, alpha_z=2.0) == golden["pi_pow10"][str(X)]   # asked for by the caller
        finally:
            ctx.close()
    with pytest.raises(pcg.PrimecountError) as e:
        pcg.Context(X, narrow - 1)
    assert e.value.status == 3


def test_budget_of_the_wide_table(pcg, golden):
    y, wide, _ = _sizes(pcg)
    ctx = pcg.Context(X, wide)
    try:
        assert ctx.table_info("factor_d")[2] == 2 * y
        assert pcg.pi(X, ctx=ctx) == golden["pi_pow10"][str(X)]
        assert ctx.table_info("factor_d")[2] == 2 * y
    finally:
        ctx.close()
