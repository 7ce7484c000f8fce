"""Rows at the global minimum and next to it, where the terms of a sum cancel: rastrigin is exactly 0 at 0, as the
reference is, and nowhere below, by every path that evaluates it; griewank is 0 at 0."""
import numpy as np
import pytest

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import archipelago as A
from pagmo2_gb300 import batch_evaluators as B
from pagmo2_gb300 import problems as P
from pagmo2_gb300.algorithms import gpu_mbh

pytestmark = pytest.mark.gpu

DIMS = [1, 2, 10, 50, 333, 1000, 1025]


def small_rows(dim, n=64):
    rng = np.random.default_rng(dim)
    x = rng.uniform(-1, 1, (n, dim)) * 10.0 ** rng.uniform(-16, -1, (n, 1))
    x[0] = 0.0
    x[1] = -0.0
    x[2] = 2.0 ** -1074
    x[3] = -1e-12
    return x


@pytest.mark.parametrize("dim", DIMS)
def test_rastrigin(ctx, dim):
    x = small_rows(dim)
    udp = P.from_kind(N.RASTRIGIN, dim, ctx)
    f = udp.batch_fitness(x)
    fg, _ = udp.batch_gradient(x)
    assert np.array_equal(f, fg)
    assert np.all(f[:3] == 0.0) and np.all(f >= 0.0)
    bfe = B.bfe(B.gpu_bfe())
    assert np.array_equal(bfe(B.problem(P.from_kind(N.RASTRIGIN, dim)), x.reshape(-1)), f)


def test_rastrigin_epoch(ctx):
    shapes = [(N.RASTRIGIN, dim, 64, grad) for dim in DIMS for grad in (False, True)]
    batches = [small_rows(dim) for _, dim, _, _ in shapes]
    ep = A.Epoch(shapes, ctx)
    try:
        for (f, _), x in zip(ep.run(batches), batches):
            assert np.all(f[:3] == 0.0) and np.all(f >= 0.0)
    finally:
        ep.close()


@pytest.mark.parametrize("dim", [2, 50, 333])
def test_rastrigin_refined(ctx, dim):
    # the minimum is where no refinement improves
    x, f, _ = gpu_mbh(hops=2, stop=2, steps=4, perturb=0.01, seed=3, context=ctx).refine(
        P.from_kind(N.RASTRIGIN, dim, ctx), np.zeros((8, dim)))
    assert np.all(f == 0.0) and np.all(x == 0.0)


@pytest.mark.parametrize("dim", DIMS)
def test_griewank(ctx, dim):
    f = P.from_kind(N.GRIEWANK, dim, ctx).batch_fitness(small_rows(dim))
    assert np.all(f[:3] == 0.0)


@pytest.mark.parametrize("dim", DIMS)
@pytest.mark.parametrize("e", [-300, -40, -30, -26, -20, -17, -16, -15])
def test_griewank_next_to_zero(ctx, dim, e):
    # |x| around 2^e, over the end of the table's range (2^-16), some elements 0: three roundings next to 1 (2^-54 each)
    # and three units of 2^-62 per factor; nowhere below 0
    rng = np.random.default_rng(dim - e)
    x = np.ldexp(rng.uniform(0.25, 1.0, (200, dim)), e + 1) * rng.choice([-1.0, 0.0, 1.0], (200, dim), p=[0.45, 0.1, 0.45])
    f = P.from_kind(N.GRIEWANK, dim, ctx).batch_fitness(x)
    z = np.longdouble(1) * x * x
    k = np.arange(1, dim + 1) * np.longdouble(1)
    want = z.sum(axis=1) / 4000 - np.expm1(np.log1p(-(z / k / 2 - (z / k) ** 2 / 24)).sum(axis=1))
    assert np.all(f >= 0.0)
    assert np.all(np.abs(f - want) <= 3 * 2.0 ** -54 + 3 * dim * 2.0 ** -62 + np.abs(want) * 2.0 ** -52)
