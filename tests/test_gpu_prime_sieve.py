"""The prime sieve's segment sizes: pi(x) counted by the sieve (a context
without tables) around the lengths where the segment changes, from one segment
of the smallest size to full ones, against the oracle's sieve; several threads
with different sizes at once."""
import threading

import pytest

pytestmark = pytest.mark.gpu

WORD, SMALL, FULL = 240, 256 * 240, 12288 * 240


def _xs():
    xs = [6, 7, 66, 67, 66 * 66, 67 * 67, 67 * 67 - 1]
    for base in (WORD, SMALL, 2 * SMALL, 300 * SMALL, 304 * SMALL, 330 * SMALL, FULL, 31 * FULL):
        xs += [base - 2, base - 1, base, base + 1, base + 17]
    return xs


def test_sieve_sizes(pcg, ora):
    ctx = pcg.Context(0)
    for x in _xs():
        assert pcg.pi(x, ctx=ctx) == ora.pi_sieve(x), x
    ctx.close()


def test_sieve_sizes_in_threads(pcg, ora):
    # calls of different segment sizes share the kernel's launch attributes
    xs = [10 ** 4 + 7, 10 ** 6 + 7, 10 ** 7 + 7, 3 * 10 ** 8 + 7]
    want = {x: ora.pi_sieve(x) for x in xs}
    bad = []

    def work(x):
        ctx = pcg.Context(0)
        for _ in range(60):
            if pcg.pi(x, ctx=ctx) != want[x]:
                bad.append(x)
        ctx.close()

    th = [threading.Thread(target=work, args=(x,)) for x in xs * 2]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
