"""phi(x, a) on both sides of the line between its leaves and P2 + P3:
phi(x, a - 1) - phi(x, a) = phi(x / p_a, a - 1) with a counted from both sides,
and the same across a wide step of a within the leaves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _primes(n):
    s = np.ones(n + 1, dtype=bool)
    s[:2] = False
    for p in range(2, int(n ** 0.5) + 1):
        if s[p]:
            s[p * p::p] = False
    return np.nonzero(s)[0]


@pytest.mark.parametrize("x", [10 ** 9 + 7, 123456789012, 10 ** 13 - 1, 98765432101234, 10 ** 15 + 3,
                               10 ** 16 - 61, 10 ** 17 + 1])
def test_line(pcg, x):
    primes = _primes(400000)
    ctx = pcg.Context(x)
    try:
        line = min(380000.0, max(50000.0 * (x / 1e15) ** 0.35, x ** 0.25))
        a0 = int(np.searchsorted(primes, line, side="right"))        # the last a by leaves, or one off
        for a in range(a0 - 2, a0 + 3):
            p = int(primes[a - 1])
            assert pcg.phi(x, a - 1, ctx=ctx) - pcg.phi(x, a, ctx=ctx) == pcg.phi(x // p, a - 1, ctx=ctx), a
        # from a to a + 40 within the leaves (y differs with a)
        for a in (9, a0 // 3 + 9):
            d = sum(pcg.phi(x // int(primes[b]), b, ctx=ctx) for b in range(a, a + 40))
            assert pcg.phi(x, a, ctx=ctx) - pcg.phi(x, a + 40, ctx=ctx) == d, a
    finally:
        ctx.close()
