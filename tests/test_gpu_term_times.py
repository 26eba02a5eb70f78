"""The times of pi(x)'s terms (pcg_stats ac_ms, b_ms, phi0_ms, sigma_ms, d_ms):
each is its own term's time, and kernel_launches counts the launches made."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TERMS = ("ac_ms", "b_ms", "phi0_ms", "sigma_ms", "d_ms")


@pytest.mark.parametrize("x", [10 ** 11, 10 ** 13, 10 ** 15, 10 ** 18])
def test_every_term_has_a_time(pcg, golden, x):
    ctx = pcg.Context(x)
    try:
        for _ in range(2):
            assert pcg.pi(x, ctx=ctx) == golden["pi_pow10"][str(x)]
        s = ctx.last_stats()
        for t in TERMS:
            assert 0 < s[t] <= s["total_ms"], (t, s)
        # D runs beside the other four, which follow one another on one stream
        assert sum(s[t] for t in TERMS[:4]) <= s["total_ms"], s
    finally:
        ctx.close()


def test_terms_one_after_another():
    # nothing overlaps: the times add up to the call, and A + C, whose pair sums are
    # listed in several batches at 1e20, outweighs B, which outweighs Phi0 and Sigma
    code = ("import primecount_gb300 as p\n"
            "for x in (10 ** 18, 10 ** 20):\n"
            "    c = p.Context(x); p.pi(x, ctx=c); p.pi(x, ctx=c); s = c.last_stats(); c.close()\n"
            "    t = [s[k] for k in %r]\n"
            "    print(x, s['total_ms'], *t)\n" % (TERMS,))
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, PCG_PI_OVERLAP="0"),
                         capture_output=True, text=True, check=True).stdout
    rows = [[float(v) for v in l.split()] for l in out.splitlines()]
    assert len(rows) == 2
    for x, total, ac, b, phi0, sigma, d in rows:
        assert 0.8 * total <= ac + b + phi0 + sigma + d <= 1.05 * total, out
        assert ac > b > phi0 > 0 and b > sigma > 0, out


@pytest.mark.parametrize("x", [10 ** 11, 10 ** 12])
def test_launches_counted(pcg, x):
    # pi(x) of one sweep wave and pair sums without pieces: k_sweep, k_combine, k_psieve, k_phi0,
    # k_sigma, and the outers of A, C1, C2 (and C1's products) that have any, and their sum
    ctx = pcg.Context(x)
    try:
        pcg.pi(x, ctx=ctx)
        pcg.pi(x, ctx=ctx)
        s = ctx.last_stats()
        p = pcg.gourdon_params(x)
        primes = [int(q) for q in ctx.read_table("primes")[1:]]
        count = lambda v: sum(1 for q in primes if q <= v)
        root = lambda v, n: max(r for r in range(int(v ** (1.0 / n)) - 2, int(v ** (1.0 / n)) + 3) if r ** n <= v)
        y, z, k, xs = p["y"], p["z"], p["k"], p["x_star"]
        sz = count(root(z, 2))
        a = count(root(x, 3)) - count(xs)
        c1 = sz - max(k, count(root(x // z, 3)))
        c2 = count(xs) - max(k, count(root(x // y, 3)), sz)
        outers = [a > 0, c1 > 0, c2 > 0]
        low = 2 * s["sweep_launches"] + 3 + sum(outers) + 1
        assert low <= s["kernel_launches"] <= low + (1 if c1 > 0 else 0), (s, a, c1, c2)
    finally:
        ctx.close()
