"""P3 of phi(x, a) just past the line between its leaves and P2 + P3, where x is
so large that its pairs' n = x / (p q) reach past the first segment of the pair
sums: phi(x, a) - phi(x, a + 1) = phi(x / p, a), p the (a + 1)-th prime."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEGMENT = 13312 * 120       # numbers per segment of the pair sums


@pytest.mark.parametrize("x", [2 * 10 ** 17 + 3, 27 * 10 ** 16 + 1])
def test_third_term_past_the_first_segment(pcg, x):
    s = np.ones(700000, dtype=bool)
    s[:2] = False
    for q in range(2, 837):
        if s[q]:
            s[q * q::q] = False
    primes = np.nonzero(s)[0]
    line = 50000.0 * (x / 1e15) ** 0.35
    assert line < 380000
    a = int(np.searchsorted(primes, line, side="right"))        # p_a <= line < p_{a + 1}
    pa, p1, p2 = (int(primes[a + i]) for i in (-1, 0, 1))
    assert pa <= line < p1 and p2 ** 3 < x and p2 ** 4 > x
    assert x // (p2 * p2) > SEGMENT and 2 * int(x ** 0.5) < 1 << 30
    ctx = pcg.Context(0)
    try:
        by_leaves = pcg.phi(x, a, ctx=ctx)
        for i in range(3):                                       # by P2 + P3
            q = int(primes[a + i])
            by_leaves -= pcg.phi(x // q, a + i, ctx=ctx)
            assert pcg.phi(x, a + 1 + i, ctx=ctx) == by_leaves, i
    finally:
        ctx.close()
