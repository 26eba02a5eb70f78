"""Levels answered in groups (k_sweep): the sums against the oracle for segment
sizes from one mask word per level to the longest levels, CTA widths, k below
the pattern primes, and group sizes around the warp and batch edges."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(2048, 128), (2048, 256), (6144, 256), (8192, 256), (10240, 256), (16384, 512), (20480, 256)]
XS = [3 * 10 ** 9 + 17, 777777777777, 23456789012345]


@pytest.mark.parametrize("x", XS)
def test_groups_against_oracle(pcg, ora, x):
    p, d = pcg.gourdon_params(x), pcg.dr_params(x)
    for k in (p["k"], 0, 2):
        want = ora.D(x, p["y"], p["z"], k, threads=8)[0]
        for words, nt in SHAPES:
            assert pcg.D(x, p["y"], p["z"], k, segment_words=words, cta_threads=nt) == want, (k, words, nt)
    want = ora.S2_hard(x, d["y"], d["z"], d["c"], threads=8)[0]
    for words, nt in SHAPES:
        assert pcg.S2_hard(x, d["y"], d["z"], d["c"], segment_words=words, cta_threads=nt) == want, (words, nt)


@pytest.mark.parametrize("group", [0, 2, 31, 33, 255])
def test_group_sizes(pcg, ora, group):
    # the group limit is read once per process
    want = [ora.D(x, *[pcg.gourdon_params(x)[n] for n in ("y", "z", "k")], threads=8)[0] for x in XS]
    code = "import primecount_gb300 as p; print(*[p.D_default(x) for x in %r])" % (XS,)
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, PCG_SWEEP_GROUP=str(group)),
                         capture_output=True, text=True, check=True).stdout
    assert [int(v) for v in out.split()] == want
