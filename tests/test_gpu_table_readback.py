"""pcg_ctx_read_table of the FactorTable: the entries for the y that the table was
built with, whatever y the calls since then have had, and calls after a read."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

X = 10 ** 17


@pytest.mark.parametrize("wide", [False, True])
def test_readback_after_other_y(pcg, ora, wide):
    if wide:
        os.environ["PCG_FACTOR_D_U32"] = "1"
    try:
        y, k = pcg.gourdon_params(X)["y"], 8
        ctx, ref = pcg.Context(X), pcg.Context(0)
        n, eb, lim = ctx.table_info("factor_d")
        assert (eb, lim) == (4 if wide else 2, 2 * y)
        built = ctx.read_table("factor_d")
        want = np.array(ora.factor_table_d16(y, 2 * y), dtype=built.dtype)
        if wide:
            want = np.where(want >= 0xFFFE, want + np.uint32(0xFFFF0000), want)
        assert np.array_equal(built, want)
        calls = [(X, y, y, k), (X - 1, y // 2, y, k), (X, y // 3, 2 * y, k), (10 ** 15, y // 7, y // 7, k)]
        for c in calls + calls[::-1]:
            want_d = pcg.D(*c, ctx=ref)
            assert pcg.D(*c, ctx=ctx) == want_d, c
            assert ctx.table_info("factor_d") == (n, eb, lim)
            assert np.array_equal(ctx.read_table("factor_d"), built), c
            assert pcg.D(*c, ctx=ctx) == want_d, c          # and the same call after the read
            out = pcg.I128()
            st = pcg.load().pcg_D_noalloc(ctx._h, pcg.to_i128(c[0]), ctypes.c_int64(c[1]), ctypes.c_int64(c[2]),
                                          ctypes.c_int64(c[3]), None, ctypes.byref(out))
            assert st == 0 and pcg.from_i128(out) == want_d, c
            assert np.array_equal(ctx.read_table("factor_d"), built), c
        ctx.close()
        ref.close()
    finally:
        if wide:
            del os.environ["PCG_FACTOR_D_U32"]


def test_part_of_the_table(pcg):
    # a read of some entries on their own, after a call with a smaller y
    y = pcg.gourdon_params(X)["y"]
    ctx = pcg.Context(X)
    built = ctx.read_table("factor_d")
    for first, count in ((0, 1), (len(built) // 2 - 700, 1400), (len(built) - 1, 1)):
        pcg.D(X, y // 3, 2 * y, 8, ctx=ctx)
        assert np.array_equal(ctx.read_table("factor_d", first, count), built[first:first + count])
    ctx.close()
