"""pi_batch: queries on both sides of the size from which they are computed whole."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [10 ** 10, 3 * 10 ** 14])
def test_both_sides(pcg, edge):
    xs = [edge - 1, edge, edge + 1, edge // 3, 2 * edge, 10 ** 6, 0]
    ctx = pcg.Context(2 * edge)
    try:
        assert pcg.pi_batch(xs, ctx=ctx) == [pcg.pi(x, ctx=ctx) for x in xs]
        assert pcg.pi_batch(xs[:2] * 5, ctx=ctx) == [pcg.pi(x) for x in xs[:2]] * 5
    finally:
        ctx.close()
