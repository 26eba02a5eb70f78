"""pi(x) by the other formula's entry point for x <= 1e10 is a sieve's count on
every context: no table of Gourdon's formula is read or built for it, so it
stays a second opinion where pi(x) itself takes the formula."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x", [1200000000, 5 * 10 ** 9 + 11, 10 ** 10])
def test_sieve_on_a_context_with_tables(pcg, x):
    ctx = pcg.Context(10 ** 12)
    try:
        before = ctx.device_bytes()
        got = pcg.pi_deleglise_rivat(x, ctx=ctx)
        # the sieve's results of 24 bytes per 12288 words; the formula's table of phi(n, k) alone has 2.4 MB
        assert ctx.device_bytes() - before < 1 << 20
        assert got == pcg.pi(x, ctx=ctx)
    finally:
        ctx.close()
