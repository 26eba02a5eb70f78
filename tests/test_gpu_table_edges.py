"""GPU: the prime tables and FactorTables at the edges of their blocks, entry by
entry: limits of one block, of a block per SM, of 2048 words a block; z at a
turn of the 2310 wheel and at a block of 8 turns, with y far below z too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1000, 1200, 128 * 240 - 2, 128 * 240, 128 * 240 + 2, 4669438, 4669442, 7777776,
                                   2048 * 152 * 240 + 12])
def test_prime_tables(pcg, limit):
    s = np.ones(limit + 1, dtype=bool)
    s[:2] = False
    for p in range(2, int(limit ** 0.5) + 1):
        if s[p]:
            s[p * p::p] = False
    want = np.nonzero(s)[0]
    ctx = pcg.Context(0)
    try:
        pcg.phi(((limit - 10) // 2) ** 2, 9, ctx=ctx)        # tables to 2 sqrt(x) + 10
        assert ctx.table_info("pi")[2] == limit
        got = ctx.read_table("primes")
        assert np.array_equal(got[1:1 + len(want)], want)
        pi = ctx.read_table("pi").reshape(-1, 2)
        starts = np.arange(len(pi), dtype=np.int64) * 240
        before = np.searchsorted(want, starts[1:])          # primes below each word
        assert np.array_equal(pi[1:, 0].astype(np.int64), before)
    finally:
        ctx.close()


@pytest.mark.parametrize("z", [2309, 2310, 2311, 18479, 18480, 18481, 18480 * 153 + 13, 777777])
@pytest.mark.parametrize("part", [1, 2, 40])
def test_factor_tables(pcg, ora, z, part):
    y = max(z // part, 60)
    ctx = pcg.Context(0)
    try:
        pcg.D(y * z, y, z, 4, ctx=ctx)
        got = ctx.read_table("factor_d")
        want = np.array(ora.factor_table_d16(y, z), dtype=np.uint16)
        assert np.array_equal(got, want), np.nonzero(got != want)[0][:5]
        if part == 1:
            pcg.S2_hard(y * z, y, z, 4, ctx=ctx)
            got = ctx.read_table("factor_dr")
            want = np.array(ora.factor_table_dr16(y), dtype=np.uint16)
            assert np.array_equal(got, want), np.nonzero(got != want)[0][:5]
    finally:
        ctx.close()
