"""pi(x) of 1.2e9 <= x <= 1e10: by Gourdon's formula on a context that holds its
tables, by the sieve on one that does not; the two agree, also through batches
and after phi has replaced the context's FactorTable."""
import random

import pytest

pytestmark = pytest.mark.gpu


def test_formula_equals_sieve(pcg):
    rng = random.Random(11)
    xs = [1199999999, 1200000000, 1200000001, 9999999999, 10000000000, 10000000001]
    xs += [int(10 ** rng.uniform(9.0792, 10)) for _ in range(60)]
    sieve, formula = pcg.Context(0), pcg.Context(10 ** 10 + 10)
    want = [pcg.pi(x, ctx=sieve) for x in xs]
    assert [pcg.pi(x, ctx=formula) for x in xs] == want
    assert pcg.pi_batch(xs, ctx=formula) == want
    pcg.phi(9 * 10 ** 9, 40, ctx=formula)          # its FactorTable is limited to p_40
    assert [pcg.pi(x, ctx=formula) for x in xs[:8]] == want[:8]
    sieve.close()
    formula.close()
