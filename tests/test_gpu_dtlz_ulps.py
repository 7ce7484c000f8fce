"""DTLZ's sines and cosines to the last place, against extended precision: with x_M = 0.5 the distance is 0 and DTLZ2's
two objectives are the cosine and the sine of fl(x fl(pi/2)) themselves. (The tests by error scale cannot see what a
fixed-point value loses where it is small.)"""
import numpy as np
import pytest

from pagmo2_gb300 import problems as P

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.mark.parametrize("e", list(range(-30, -9, 4)) + list(range(-9, 1)))
@pytest.mark.parametrize("side", ["sine", "cosine"])
def test_dtlz2(ctx, e, side):
    if np.finfo(LD).nmant < 63:
        pytest.skip("needs a long double beyond double")
    rng = np.random.default_rng(e + 50)
    t = np.ldexp(rng.uniform(0.5, 1.0, 20000), e)
    x = np.full((20000, 6), 0.5)
    x[:, 0] = t if side == "sine" else 1.0 - t
    f = P.dtlz(2, 6, 2, 100, ctx).batch_fitness(x).reshape(-1, 2)
    y = LD(1) * (x[:, 0] * (np.pi / 2))
    # a value from the table: its 2^-60 and one rounding; below 2^-6 the series' last step, the cosine's angle too
    for got, want in ((f[:, 0], np.cos(y)), (f[:, 1], np.sin(y))):
        rel = np.where(np.abs(want) < 2.0 ** -6, LD(2) ** -52, LD(2) ** -53)
        bound = np.abs(want) * rel + np.where(np.abs(want) < 2.0 ** -6, 0, LD(2) ** -60)
        assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))


@pytest.mark.parametrize("scale", [0.5, 1e-2, 1e-5, 1e-8])
def test_distance_is_not_biased(ctx, scale):
    # x_0 = 0: the first objective is 1 + g, g the sum of ten squares. One rounding, uniform within 2^-53 where g spreads
    # over many units of 2^-52 and is below 1: the mean of 400000 errors lies within 5 deviations of 0, 2^-53 /
    # sqrt(3 * 400000) each; the squares' own errors are below a hundredth of that rounding. (At 1e-8 g is of the size
    # of one unit, and the correctly rounded values' errors have a mean of -1.2e-18 themselves.)
    if np.finfo(LD).nmant < 63:
        pytest.skip("needs a long double beyond double")
    n = 400000
    rng = np.random.default_rng(11)
    x = 0.5 + scale * (2.0 * rng.random((n, 11)) - 1.0)
    x[:, 0] = 0.0
    if scale == 0.5:
        x[:, 4:] = 0.5 + 0.2 * (2.0 * rng.random((n, 7)) - 1.0)
    f = P.dtlz(2, 11, 2, 100, ctx).batch_fitness(x).reshape(-1, 2)[:, 0]
    want = 1 + ((LD(1) * x[:, 1:] - LD(0.5)) ** 2).sum(axis=1)
    e = (f - want).astype(float)
    assert np.max(np.abs(e)) <= 2.0 ** -53 * 1.01 * (1 if scale < 0.5 else 2)
    if scale in (1e-2, 1e-5):
        assert abs(e.mean()) <= 5 * 2.0 ** -53 / np.sqrt(3 * n)
