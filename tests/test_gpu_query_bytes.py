"""pcg_query_device_bytes is at or above the device memory that the call takes
beyond the context's resident tables: contexts without tables, made for the
query, and made for a far larger one."""
import math

import pytest

pytestmark = pytest.mark.gpu

PIS = [10 ** 3, 10 ** 6, 5 * 10 ** 8, 1200000000, 5 * 10 ** 9, 10 ** 10, 10 ** 10 + 1, 3 * 10 ** 10, 10 ** 11, 10 ** 12,
       10 ** 13, 10 ** 14, 3 * 10 ** 14, 10 ** 15, 10 ** 16, 3 * 10 ** 16, 10 ** 17, 10 ** 18, 10 ** 19]


def _grown(ctx, call):
    ctx.trim()
    before = ctx.device_bytes()
    call()
    return ctx.device_bytes() - before


@pytest.mark.parametrize("made_for", ["none", "query", "large"])
def test_pi(pcg, made_for):
    low = []
    for x in PIS:
        ctx = pcg.Context({"none": 0, "query": x, "large": 10 ** 19}[made_for])
        for turn in range(2):                    # the first call also builds tables of its own
            est = pcg.query_device_bytes("pi", x, ctx=ctx)
            got = _grown(ctx, lambda: pcg.pi(x, ctx=ctx))
            if got > est:
                low.append((x, turn, got, est))
        ctx.close()
    assert not low


@pytest.mark.parametrize("made_for", ["none", "query", "large"])
def test_phi(pcg, made_for):
    low = []
    for x in [10 ** 6, 10 ** 8 + 7, 2 * 10 ** 9, 10 ** 11, 10 ** 13, 10 ** 14, 10 ** 16, 4 * 10 ** 17]:
        sq = math.isqrt(x)
        top = sq / math.log(sq)
        line = 50000.0 * (x / 1e15) ** 0.35
        marks = [2, 8, 9, 40, x ** 0.25 / math.log(x ** 0.25), 0.97 * line / math.log(max(line, 3)),
                 1.1 * line / math.log(max(line, 3)), x ** (1 / 3) / math.log(x ** (1 / 3)), 0.5 * top, 1.2 * top]
        for a in sorted({max(2, int(v)) for v in marks}):
            ctx = pcg.Context({"none": 0, "query": x, "large": 10 ** 19}[made_for])
            for turn in range(2):
                est = pcg.query_device_bytes("phi", x, a, ctx=ctx)
                got = _grown(ctx, lambda: pcg.phi(x, a, ctx=ctx))
                if got > est:
                    low.append((x, a, turn, got, est))
            ctx.close()
    assert not low
