"""The work that users have this framework do, through its public entry points.

Every case is one pass of one kind of call ("call"), at a size ("x", "n"); the
seed perturbs x by up to 1/64 downwards, so sizes are odd and ragged and no two
seeds give the same inputs.  All results are exact integers: run() returns them
as rows of two int64 words (the low 62 bits and the rest).
"""
import math
import random

import numpy as np

import primecount_gb300 as pcg

MASK62 = (1 << 62) - 1


def listed():
    return [
        # the smallest call: one pi(x) of a few million, where launches and copies count
        {"name": "pi_1e6", "call": "pi", "x": 10 ** 6},
        # pi(x) below 1e10, the everyday range of the command line
        {"name": "pi_5e9", "call": "pi", "x": 5 * 10 ** 9},
        # pi(x) on a kept context (a program asking again and again): small, ...
        {"name": "pi_1e13", "call": "pi", "x": 10 ** 13},
        # ... ordinary, ...
        {"name": "pi_1e18", "call": "pi", "x": 10 ** 18},
        # ... and large (x above 2^64)
        {"name": "pi_2e19", "call": "pi", "x": 2 * 10 ** 19},
        # a one-shot call, tables built inside it: what `python -m primecount_gb300 1e16` does
        {"name": "pi_1e16_once", "call": "pi_once", "x": 10 ** 16},
        # pi(x) by the other formula the framework offers (option -d)
        {"name": "pi_dr_1e16", "call": "pi_dr", "x": 10 ** 16},
        # the hard special leaves alone (option --D): a small one ...
        {"name": "D_1e15", "call": "D", "x": 10 ** 15},
        # ... and the headline size of the benchmark
        {"name": "D_1e20", "call": "D", "x": 10 ** 20},
        # Deleglise-Rivat's hard special leaves (option --S2-hard)
        {"name": "S2_hard_1e17", "call": "S2_hard", "x": 10 ** 17},
        # phi(x, a) one after another, a over its whole range (all the ways phi is computed)
        {"name": "phi_1e14", "call": "phi", "x": 10 ** 14, "n": 8},
        # many queries of very different sizes in one call: pi(x) and phi(x, a)
        {"name": "batch_1e16", "call": "batch", "x": 10 ** 16, "n": 32},
    ]


# call -> (smallest, largest) decimal exponent of x, as the listed cases stand for
RANGES = {"pi": (4.0, 19.3), "pi_once": (9.0, 18.0), "pi_dr": (11.0, 18.0), "D": (12.0, 19.7),
          "S2_hard": (12.0, 18.3), "phi": (9.0, 16.0), "batch": (12.0, 16.0)}


def draw(rng):
    call = rng.choice(["pi", "pi", "pi", "pi_once", "pi_dr", "D", "D", "S2_hard", "phi", "batch"])
    case = {"call": call, "x": int(10 ** rng.uniform(*RANGES[call]))}
    if call == "phi":
        case["n"] = rng.randint(3, 12)
    if call == "batch":
        case["n"] = rng.randint(6, 40)
    return case


def _below(rng, x):
    return x - rng.randrange(x // 64 + 1)


def _phi_query(rng, x):
    """An a for phi(x, a): spread over the logarithm of 2 .. 2 pi(sqrt(x))."""
    top = 2.0 * math.sqrt(x) / max(1.0, math.log(math.sqrt(x)))
    return x, int(math.exp(rng.uniform(math.log(2.0), math.log(max(3.0, top)))))


def _inputs(case, seed):
    rng = random.Random(1000003 * seed + 17)
    x, call = case["x"], case["call"]
    if call == "phi":
        # a stratified over its range, so that every seed asks for every kind of phi
        got = []
        for i in range(case["n"]):
            xi = _below(rng, x)
            top = math.log(2.0 * math.sqrt(xi) / max(1.0, math.log(math.sqrt(xi))))
            got.append((xi, int(math.exp(math.log(2.0) + (top - math.log(2.0)) * (i + rng.random()) / case["n"]))))
        return got
    if call == "batch":
        # sizes spread over the decades below x; stratified, so that seeds differ little in work
        lo, hi, n = 9.0, math.log10(x), case["n"]
        pis = [_below(rng, int(10 ** (lo + (hi - lo) * (i + 0.5) / n))) for i in range(n)]
        phis = [_phi_query(rng, _below(rng, int(10 ** (lo + (hi - lo) * (i + 0.5) / n)))) for i in range(n)]
        rng.shuffle(pis)
        rng.shuffle(phis)
        return pis, phis
    return _below(rng, x)


def prepare(case, seed):
    """The query and the context a program keeps: its tables cover x."""
    state = {"call": case["call"], "q": _inputs(case, seed), "ctx": None}
    if case["call"] != "pi_once":
        state["ctx"] = pcg.Context(case["x"])
    if case["call"] == "D":
        p = pcg.gourdon_params(state["q"])
        state["args"] = (p["y"], p["z"], p["k"])
    if case["call"] == "S2_hard":
        p = pcg.dr_params(state["q"])
        state["args"] = (p["y"], p["z"], p["c"])
    return state


def _rows(values):
    return np.array([[v & MASK62, v >> 62] for v in values], dtype=np.int64)


def run(state):
    call, q, ctx = state["call"], state["q"], state["ctx"]
    if call == "pi":
        return _rows([pcg.pi(q, ctx=ctx)])
    if call == "pi_once":
        ctx = pcg.Context()
        v = pcg.pi(q, ctx=ctx)
        ctx.close()
        return _rows([v])
    if call == "pi_dr":
        return _rows([pcg.pi_deleglise_rivat(q, ctx=ctx)])
    if call == "D":
        return _rows([pcg.D(q, *state["args"], ctx=ctx)])
    if call == "S2_hard":
        return _rows([pcg.S2_hard(q, *state["args"], ctx=ctx)])
    if call == "phi":
        return _rows([pcg.phi(x, a, ctx=ctx) for x, a in q])
    pis, phis = q
    return {"pi": _rows(pcg.pi_batch(pis, ctx=ctx)),
            "phi": _rows(pcg.phi_batch([x for x, _ in phis], [a for _, a in phis]))}


# Leaves and crossed-off multiples of the hard leaves at 10^11, 10^12, ... (the formulas' own
# counts, the same for every implementation that sieves [0, x / z) by the level).
_D_LEAVES = [8.29e4, 5.24e5, 2.22e6, 8.38e6, 3.06e7, 1.11e8, 4.08e8, 1.52e9, 5.79e9, 2.22e10]
_D_CROSS = [1.73e6, 3.63e6, 1.25e7, 4.85e7, 1.96e8, 7.86e8, 3.10e9, 1.19e10, 4.50e10, 1.68e11]


def _at(table, x):
    e = max(0.0, math.log10(max(x, 2)) - 11.0)
    i = min(int(e), len(table) - 2)
    return table[i] * (table[i + 1] / table[i]) ** (e - i)


def _d_ops(x):
    # a division and a prefix query of a counter and a word (about 10 operations) per leaf, one
    # read-modify-write per multiple
    return 10.0 * _at(_D_LEAVES, x) + _at(_D_CROSS, x)


def _sieve_ops(x):
    # 8 of 30 numbers, each crossed off about log log x times, read once for the count
    return (8.0 / 30.0) * x * (math.log(max(1.1, math.log(max(x, 20)))) + 1.0 / 64)


def _pi_ops(x):
    if x <= 10 ** 10:
        return _sieve_ops(x)
    # A + C: 2.3e11 terms at 1e20, a multiplication and a table lookup (about 6 operations) each;
    # B: the primes of [sqrt(x), x / y)
    y = pcg.gourdon_params(x)["y"]
    return _d_ops(x) + 6.0 * 2.3e11 * (x / 1e20) ** 0.66 + _sieve_ops(x // max(1, y))


def _phi_ops(x):
    # the mean over a: between the trivial forms and pi(x) with a second sieve
    return 0.5 * _pi_ops(x)


def _table_bytes(x):
    # the tables, read once: 2 bytes per number <= z coprime to 2310, 4 per prime <= y, 16 per
    # 240 numbers <= y
    if x <= 10 ** 10:
        return 64.0
    p = pcg.gourdon_params(x)
    y, z = p["y"], p["z"]
    return 2.0 * z * 480 / 2310 + 4.0 * y / math.log(y) + 16.0 * y / 240


def work(case):
    x, call = case["x"], case["call"]
    if call in ("pi", "pi_once"):
        big = 16.0 * math.isqrt(x) / 240 if x > 10 ** 10 else 0.0   # the prime counts up to sqrt(x)
        return {"bytes": _table_bytes(x) + big + 32.0, "flops": _pi_ops(x)}
    if call == "pi_dr":
        return {"bytes": _table_bytes(x) + 16.0 * math.isqrt(x) / 240 + 32.0, "flops": 1.4 * _pi_ops(x)}
    if call == "D":
        return {"bytes": _table_bytes(x) + 64.0, "flops": _d_ops(x)}
    if call == "S2_hard":
        return {"bytes": _table_bytes(x) + 64.0, "flops": 1.4 * _d_ops(x)}
    if call == "phi":
        return {"bytes": 32.0 * case["n"], "flops": case["n"] * _phi_ops(x)}
    n = case["n"]
    xs = [int(10 ** (9.0 + (math.log10(x) - 9.0) * (i + 0.5) / n)) for i in range(n)]
    return {"bytes": 64.0 * n + max(_table_bytes(v) for v in xs),
            "flops": sum(_pi_ops(v) + _phi_ops(v) for v in xs)}


def _lucy(x):
    """pi(x) for x up to about 1e11: the counts of n <= x // i left after each prime (numpy, 64 bits)."""
    if x < 2:
        return 0
    r = math.isqrt(x)
    idx = np.arange(1, r + 1, dtype=np.int64)
    small = np.arange(r + 1, dtype=np.int64) - 1       # counts for n <= r
    large = np.empty(r + 1, dtype=np.int64)            # counts for x // i
    large[1:] = x // idx - 1
    for p in range(2, r + 1):
        if small[p] == small[p - 1]:
            continue
        c = small[p - 1]
        top = min(r, x // (p * p))
        k = min(top, r // p)
        i = idx[:top]
        new = large[1:top + 1].copy()
        new[:k] -= large[i[:k] * p] - c
        if top > k:
            new[k:] -= small[x // (i[k:] * p)] - c
        large[1:top + 1] = new
        if p * p <= r:
            n = np.arange(p * p, r + 1, dtype=np.int64)
            small[p * p:] -= small[n // p] - c
    return int(large[1])


def exact(case, seed):
    """pi(x) of the small sizes by plain numpy; the others would take too long."""
    if case["call"] in ("pi", "pi_once") and case["x"] <= 10 ** 11:
        return _rows([_lucy(_inputs(case, seed))])
    return None
