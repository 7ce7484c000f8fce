"""Rastrigin rows with elements from 8 on, over the end of the integer range (2^11) to infinities: fitness and gradient
to the last places against long double, the same by every number of lanes, alone and in an epoch."""
import numpy as np
import pytest

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import archipelago as A
from pagmo2_gb300 import problems as P

pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288419716939937510582097494459")


def rows(dim, binades, n=200):
    rng = np.random.default_rng(dim + binades[1] + 100)
    x = np.ldexp(rng.uniform(0.5, 1.0, (n, dim)), rng.integers(*binades, (n, dim), endpoint=True))
    x *= rng.choice([-1.0, 1.0], x.shape)
    x[::2, : dim // 2] = rng.uniform(-5.12, 5.12, x[::2, : dim // 2].shape)
    x[0, 0], x[1, 0], x[2, 0] = 8.0, -2048.0, np.nextafter(2048.0, 0)
    return x


@pytest.mark.parametrize("dim", [1, 7, 50, 333, 1025])
@pytest.mark.parametrize("binades", [(4, 4), (3, 6), (5, 11), (-12, 11), (11, 13), (40, 60)])
def test_values(ctx, dim, binades):
    if np.finfo(LD).nmant < 63:
        pytest.skip("needs a long double beyond double")
    x = rows(dim, binades)
    f, g = P.from_kind(N.RASTRIGIN, dim, ctx).batch_gradient(x)
    r = LD(1) * (x - np.rint(x))
    s, c, a = np.sin(2 * PI * r), np.cos(2 * PI * r), LD(1) * x
    want = (a * a - 10 * c + 10).sum(axis=1)
    # one rounding, a unit of 2^-52 per element, 2^-62 of a far element's square and 2^-56 of a cosine; a row of larger
    # elements sums in FP64: an addition's rounding per element
    bound = np.abs(want) * LD(2) ** -52 * (1 if binades[1] <= 11 else dim) + dim * 2.0 ** -51
    row = np.arange(len(x))
    usual = row != 1  # (that row has a 2048)
    if binades[1] > 11:
        usual = row < 0
    bound = np.where(usual, bound, np.abs(want) * LD(2) ** -52 * dim + dim * 2.0 ** -51)
    assert np.all(np.abs(f - want) <= bound), float(np.max(np.abs(f - want) / bound))
    wg = 2 * a + 20 * PI * s
    bg = np.abs(wg) * LD(2) ** -53 + 20 * PI * (LD(2) ** -51 * np.abs(s) + LD(2) ** -60)
    assert np.all(np.abs(g - wg) <= bg), float(np.max(np.abs(g - wg) / bg))


@pytest.mark.parametrize("binades", [(4, 4), (-12, 11), (11, 13)])
def test_paths_agree(ctx, binades):
    dims = (4, 7, 50, 333)
    batches = [rows(d, binades) for d in dims]
    ep = A.Epoch([(N.RASTRIGIN, d, 200, True) for d in dims], ctx)
    try:
        for (f, g), x, d in zip(ep.run(batches), batches, dims):
            udp = P.from_kind(N.RASTRIGIN, d, ctx)
            f1, g1 = udp.batch_gradient(x)
            assert np.array_equal(f, f1) and np.array_equal(g, g1)
            assert np.array_equal(udp.batch_fitness(x), f1)
            # more rows, other lanes: each row's value is its own
            many = np.tile(x, (100, 1))
            f2, g2 = udp.batch_gradient(many)
            assert np.array_equal(f2, np.tile(f1, 100)) and np.array_equal(g2, np.tile(g1, (100, 1)))
    finally:
        ep.close()


def test_not_finite(ctx):
    x = np.full((4, 9), 9.5)
    x[0, 2], x[1, 3], x[2, 8] = np.inf, -np.inf, np.nan
    f, g = P.from_kind(N.RASTRIGIN, 9, ctx).batch_gradient(x)
    assert np.all(np.isnan(f[:3])) and np.isfinite(f[3])
    assert np.all(np.isnan(g[:3]) == ~np.isfinite(x[:3]))
