"""Numbers that two levels of a group cross off (k_sweep): the same sums whether
the list of them holds them all, a few or none, where each lane resolves its
own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
XS = [3 * 10 ** 9 + 17, 777777777777, 23456789012345, 10 ** 15]


@pytest.mark.parametrize("entries", [0, 2, 33])
def test_list_too_short(pcg, ora, entries):
    # the length in use is read once per process
    want = []
    for x in XS[:3]:
        p, d = pcg.gourdon_params(x), pcg.dr_params(x)
        want += [ora.D(x, p["y"], p["z"], p["k"], threads=8)[0], ora.S2_hard(x, d["y"], d["z"], d["c"], threads=8)[0]]
    want += [pcg.D_default(XS[3]), pcg.S2_hard_default(XS[3])]
    code = ("import primecount_gb300 as p\n"
            "for w, t in ((0, 0), (2048, 128), (20480, 512)):\n"
            "    print(*[f(x, segment_words=w, cta_threads=t) for x in %r for f in (p.D_default, p.S2_hard_default)])\n"
            % (XS,))
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT,
                         env=dict(os.environ, PCG_SWEEP_COLLISIONS=str(entries)), capture_output=True, text=True,
                         check=True).stdout
    rows = [[int(v) for v in l.split()] for l in out.splitlines()]
    assert len(rows) == 3
    for r in rows:
        assert r == want
