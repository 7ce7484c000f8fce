"""The sine rows to the last places, against extended precision. (The tests by error scale allow 1e-13 of it, which
hides what a fixed-point sine loses where it is small.)"""
import numpy as np
import pytest

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import problems as P

pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288419716939937510582097494459")


@pytest.fixture(autouse=True)
def extended():
    if np.finfo(LD).nmant < 63:
        pytest.skip("needs a long double beyond double")


def rastrigin_gradient(x):
    r = LD(1) * (x - np.rint(x))  # exact
    s = np.sin(2 * PI * r)
    return 2 * LD(1) * x + 20 * PI * s, s


@pytest.mark.parametrize("e", list(range(-40, -12, 7)) + list(range(-12, 4)))
def test_rastrigin_gradient(ctx, e):
    # 2^(e-1) <= |x| < 2^e. Rounded operations: the sine's conversion, the constant's rounding and the product (or,
    # for small x, the polynomial's last step and the product): 2^-53 each; the table's 2^-60, which may not be seen
    # where the sine itself is small.
    rng = np.random.default_rng(e + 100)
    x = np.ldexp(rng.uniform(0.5, 1.0, (200, 50)), e) * rng.choice([-1.0, 1.0], (200, 50))
    _, g = P.from_kind(N.RASTRIGIN, 50, ctx).batch_gradient(x)
    want, s = rastrigin_gradient(x)
    bound = np.abs(want) * LD(2) ** -53 + 20 * PI * (LD(2) ** -52 * np.abs(s) + (LD(2) ** -60 if e > -8 else 0))
    assert np.all(np.abs(g - want) <= bound), float(np.max(np.abs(g - want) / bound))


@pytest.mark.parametrize("at", [0.5, 1.0, 2.0, 3.5, 5.0])
def test_rastrigin_gradient_at_half_periods(ctx, at):
    # next to the sine's other zeros, where 2x stays: the table's error alone beside the last rounding
    rng = np.random.default_rng(int(10 * at))
    d = np.ldexp(rng.uniform(0.5, 1.0, (200, 50)), rng.integers(-40, -3, (200, 50))) * rng.choice([-1.0, 1.0], (200, 50))
    x = (at + d) * rng.choice([-1.0, 1.0], (200, 50))
    _, g = P.from_kind(N.RASTRIGIN, 50, ctx).batch_gradient(x)
    want, s = rastrigin_gradient(x)
    bound = np.abs(want) * LD(2) ** -53 + 20 * PI * (LD(2) ** -52 * np.abs(s) + LD(2) ** -60)
    assert np.all(np.abs(g - want) <= bound), float(np.max(np.abs(g - want) / bound))
