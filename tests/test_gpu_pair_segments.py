"""The pair sums by segments of n: pi(x) where the prime table just passes the
length that lists pieces, with y (and so every range of the easy formulas)
moved, against the other formula and the published values."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x", [60000000000007, 10 ** 14, 3 * 10 ** 14 + 1, 10 ** 15, 27182818284590452, 10 ** 17])
def test_pi_by_moved_ranges(pcg, golden, x):
    want = pcg.pi_deleglise_rivat(x)
    if str(x) in golden["pi_pow10"]:
        assert want == golden["pi_pow10"][str(x)]
    base = pcg.gourdon_params(x)["y"] / round(x ** (1 / 3))
    for f in (0.0, 0.3, 0.7, 1.9, 4.0):
        assert pcg.pi(x, alpha_y=f * base) == want, f


def test_phi_third_term(pcg):
    # P3 of phi(x, a) sums pairs as well: phi(x, a + 1) = phi(x, a) - phi(x / p, a), p the (a + 1)-th prime
    x, a = 10 ** 15 + 37, 3000
    p = [q for q in range(2, 40000) if all(q % d for d in range(2, int(q ** 0.5) + 1))][a]
    assert pcg.phi(x, a + 1) == pcg.phi(x, a) - pcg.phi(x // p, a)
