"""One FactorTableD for all the x of a context: D with y < z < 13 y from a table
of a larger y (its primes above y out), and back, against new contexts."""
import pytest

pytestmark = pytest.mark.gpu


def test_calls_in_turn_on_one_context(pcg, golden):
    ctx = pcg.Context(10 ** 17)
    xs = [10 ** 17, 31415926535897932, 99999999999999999, 10 ** 13 + 9]
    calls = []
    for x in xs:
        p = pcg.gourdon_params(x)
        y, k = p["y"], p["k"]
        calls += [(x, y, int(f * y), k) for f in (1, 1.5, 2, 6, 12.9)]
        calls += [(x, y // 2, y // 2, k), (x, y // 2, 2 * y, k)]
    calls.append((10 ** 13, 30000, 30000 * 14, 8))     # z > 13 y: a table of its own
    want = {}
    for c in calls:
        new = pcg.Context(0)
        want[c] = pcg.D(*c, ctx=new)
        new.close()
    for c in calls + calls[::-1] + calls[::3] + calls[1::2]:
        assert pcg.D(*c, ctx=ctx) == want[c], c
    ctx.close()


def test_pi_and_terms_in_turn(pcg, golden):
    ctx = pcg.Context(10 ** 17 + 5)
    want = golden["pi_pow10"]
    for _ in range(2):
        assert pcg.pi(10 ** 17, ctx=ctx) == want[str(10 ** 17)]       # z = 2 y
        assert pcg.pi_terms(10 ** 17, ctx=ctx)["pi"] == want[str(10 ** 17)]   # z = y
        assert pcg.pi(10 ** 17, ctx=ctx, alpha_z=3.0) == want[str(10 ** 17)]
        assert pcg.pi(10 ** 14, ctx=ctx) == want[str(10 ** 14)]
        assert pcg.phi(10 ** 12, 100, ctx=ctx) == pcg.phi(10 ** 12, 100)      # a table limited to p_100
        assert pcg.pi_batch([10 ** 16, 10 ** 17], ctx=ctx) == [want[str(10 ** 16)], want[str(10 ** 17)]]
    ctx.close()
