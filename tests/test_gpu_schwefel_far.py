"""Schwefel rows with elements below 2^-20 and from 512 on, alone and beside usual ones, over the ends of the integer
range (2^14) to infinities, against long double: an element's error is a few units of 2^-51, or of its own last place
where it is larger (the sine's 2^-57 and its angle's 2^-58 per unit of the root times |x|), the rest the closing sum's."""
import numpy as np
import pytest

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import problems as P

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.mark.parametrize("dim", [1, 5, 50, 1025])
@pytest.mark.parametrize("binades", [(-1080, -20), (-24, -18), (8, 11), (9, 14), (12, 17), (-30, 16)])
def test_rows(ctx, dim, binades):
    if np.finfo(LD).nmant < 63:
        pytest.skip("needs a long double beyond double")
    rng = np.random.default_rng(dim + binades[1] + 100)
    x = np.ldexp(rng.uniform(0.5, 1.0, (300, dim)), rng.integers(*binades, (300, dim), endpoint=True))
    x *= rng.choice([-1.0, 1.0], x.shape)
    x[::3, : dim // 2] = rng.uniform(-500, 500, x[::3, : dim // 2].shape)
    x[0, 0] = 0.0
    x[1, 0] = -512.0
    x[2, 0] = 16384.0
    f = P.from_kind(N.SCHWEFEL, dim, ctx).batch_fitness(x)
    a = LD(1) * np.abs(x)
    constant = LD(418.9828872724338) * dim
    want = constant - (x * np.sin(np.sqrt(a))).sum(axis=1)
    each = 2.0 ** -49 + a * (LD(2) ** -50 + np.sqrt(a) * LD(2) ** -53)  # (from 2^14 on the root and the sine in FP64)
    bound = each.sum(axis=1) + (constant + np.abs(want)) * LD(2) ** -52
    assert np.all(np.abs(f - want) <= bound), float(np.max(np.abs(f - want) / bound))


def test_not_finite(ctx):
    x = np.full((4, 7), 3.0)
    x[0, 2], x[1, 3], x[2, 6] = np.inf, -np.inf, np.nan
    f = P.from_kind(N.SCHWEFEL, 7, ctx).batch_fitness(x)
    assert np.all(np.isnan(f[:3])) and np.isfinite(f[3])
