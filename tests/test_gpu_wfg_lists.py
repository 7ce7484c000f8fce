"""WFG where the rows of a level outgrow its list (n^2 rows for small sets): what follows the last frame that fits holds
nothing of earlier calls. Calls of one context, large and small in turn, equal the oracle's bit for bit."""
import numpy as np
import pytest

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import multi_objective as MO

pytestmark = pytest.mark.gpu


def front(n, m, rng):
    w = rng.random((n, m)) ** 2
    return w / np.linalg.norm(w, axis=1, keepdims=True)


@pytest.mark.parametrize("m", [6, 7, 9])
def test_lists_that_overflow(orc, m):
    rng = np.random.default_rng(m)
    r = np.full(m, 1.25)
    sets = [front(n, m, rng) for n in ((60, 24, 60, 40, 57, 33) if m < 9 else (30, 20, 30, 26))]
    want = [(orc.hvwfg(p, r), orc.hvwfg_contributions(p, r)) for p in sets]
    with N.Context(0) as ctx:
        for _ in range(2):
            for p, (v, c) in zip(sets, want):
                assert MO.hypervolume(p, context=ctx).compute(r) == v
                assert np.array_equal(MO.hypervolume(p, context=ctx).contributions(r), c)


def test_large_then_small(orc):
    # a list of 2^20 rows filled by one call, then calls that share its layout or part of it
    rng = np.random.default_rng(1)
    r = np.full(6, 1.25)
    with N.Context(0) as ctx:
        MO.hypervolume(front(1500, 6, rng), context=ctx).compute(r)
        for n in (1500, 1490, 30):
            p = front(n, 6, rng)
            p[:, 3:] = np.round(p[:, 3:] * 4) / 4  # smaller limit sets
            p = p[rng.permutation(n)]
            got = MO.hypervolume(p, context=ctx).compute(r)
            if n == 30:
                assert got == orc.hvwfg(p, r)
            else:
                with N.Context(0) as fresh:
                    assert got == MO.hypervolume(p, context=fresh).compute(r)
