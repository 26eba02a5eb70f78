"""The single-precision quotient of the leaf offsets (quot_f32 in
csrc/dev_common.cuh; leaf_narrow and leaf_wide in csrc/sweep.cu), restated in numpy with the reciprocal one unit
in the last place off in either direction (its documented error): the quotient
is off by at most the corrections that follow it, so the offset is exact."""
import numpy as np
import pytest

F = np.float32


def quotient(r, m, ulp):
    inv = (F(1) / m.astype(F)).astype(F)
    if ulp:
        inv = np.nextafter(inv, F(np.inf) if ulp > 0 else F(0)).astype(F)
    hi, lo = (r >> np.uint64(32)).astype(F), (r & np.uint64(0xFFFFFFFF)).astype(F)
    # the fused multiply-add rounds once: both products fit double precision
    rf = (hi.astype(np.float64) * 4294967296.0 + lo.astype(np.float64)).astype(F)
    return np.floor((rf * inv).astype(F)).astype(np.int64)


@pytest.mark.parametrize("span,mmax,most", [(1 << 21, 1 << 30, 1), (1 << 23, 1 << 32, 3)])
@pytest.mark.parametrize("ulp", [-1, 0, 1])
def test_quotient_error(span, mmax, most, ulp):
    rng = np.random.default_rng(5)
    n = 400000
    m = np.exp(rng.uniform(0, np.log(mmax - 1), n)).astype(np.uint64)
    m = np.clip(m, 1, mmax - 1)
    m[: n // 8] = mmax - 1 - rng.integers(0, 1000, n // 8).astype(np.uint64)
    d = np.floor(np.exp(rng.uniform(0, np.log(span), n))).astype(np.uint64)
    d[::3] = span - 1 - rng.integers(0, 50, d[::3].size).astype(np.uint64)
    d = np.minimum(d, span - 1)
    t = (rng.random(n) * m.astype(np.float64)).astype(np.uint64)
    t[::5] = 0
    t[1::5] = m[1::5] - np.uint64(1)
    t = np.minimum(t, m - np.uint64(1))
    r = d * m + t                       # floor(r / m) = d
    err = quotient(r, m, ulp) - d.astype(np.int64)
    assert np.abs(err).max() <= most
    if most == 1:
        # the 32-bit remainder of the narrow form keeps its sign
        rem = r.astype(np.int64) - (d.astype(np.int64) + err) * m.astype(np.int64)
        assert np.abs(rem).max() < 1 << 31
