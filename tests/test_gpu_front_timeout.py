"""Failure detection without a fault in the two-objective survival pass: waits limited to so few polls that they give
up. The pass returns, a device caller reads -1 fronts (0 would be an empty result), nothing after it works on what the
fronts left, and the same context then runs a full pass."""
import ctypes as C

import numpy as np
import pytest

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import multi_objective as MO

pytestmark = pytest.mark.gpu


def fronts(ctx, p, limit):
    nf = C.c_int32(12345)
    N.check(N.lib().pgx_selftest_front_timeout(ctx.handle, p.ctypes.data, len(p), limit, C.byref(nf)))
    return nf.value


@pytest.mark.parametrize("n", [5000, 20000, 32768])
def test_waits_are_bounded(ctx, orc, n):
    rng = np.random.default_rng(n)
    p = np.ascontiguousarray(rng.random((n, 2)) + np.arange(n)[:, None] % 7)
    want = orc.fnds(p, dom_list=False)
    full = len(want["front_offsets"]) - 1
    assert fronts(ctx, p, 1 << 22) == full
    assert fronts(ctx, p, 1) == -1
    rank, _, off, idx, _ = MO.nsga2_survival(p, ctx)
    assert np.array_equal(rank, want["rank"])
    assert np.array_equal(off, want["front_offsets"]) and np.array_equal(idx, want["front_indices"])


def test_limits_are_checked(ctx):
    p = np.zeros((2000, 2))
    nf = C.c_int32()
    for n, limit in ((1024, 1), (32769, 1), (2000, 0), (2000, 1 << 25)):
        with pytest.raises(ValueError):
            N.check(N.lib().pgx_selftest_front_timeout(ctx.handle, p.ctypes.data, n, limit, C.byref(nf)))
