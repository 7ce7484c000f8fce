"""Infinite coordinates and reference points in the 2- and 3-objective hypervolume, which hypervolume's checks accept:
the measure of the dominated region, a side of no length making a cell empty whatever the other sides are. The oracle
(the reference's operations) gives that measure too wherever it does not form 0 * inf or inf - inf."""
import itertools

import numpy as np
import pytest

from pagmo2_gb300 import multi_objective as MO

INF = np.inf


def measure(p, r):
    """Sum over the cells of the grid of all coordinates (no cell has a side of no length)."""
    cuts = [np.unique(np.append(p[:, c], r[c])) for c in range(len(r))]
    total = 0.0
    for cell in itertools.product(*[range(len(c) - 1) for c in cuts]):
        low = np.array([c[i] for c, i in zip(cuts, cell)])
        if np.any(np.all(p <= low, axis=1)):
            total += np.prod([c[i + 1] - c[i] for c, i in zip(cuts, cell)])
    return total


def cases(m, k):
    rng = np.random.default_rng(m)
    while k:
        r = rng.choice([2.0, INF], m)
        p = np.array([[rng.choice([v for v in (-INF, 0.0, 1.0, INF) if v <= r[c]]) for c in range(m)]
                      for _ in range(rng.integers(1, 6))])
        if np.any(np.all(p == r, axis=1)):
            continue
        k -= 1
        yield p, r


@pytest.mark.parametrize("m", [2, 3])
def test_measure_is_the_oracles(orc, m):
    compared = 0
    for p, r in cases(m, 1000):
        v = orc.hypervolume(p, r)
        if not np.isnan(v):
            assert v == measure(p, r), (p, r)
            compared += 1
    assert compared > 200


@pytest.mark.gpu
@pytest.mark.parametrize("p,r,want", [([(INF, 0, 0), (INF, 1, 1)], (INF, 2, 2), 0.0),
                                      ([(INF, 0, 0), (0, 1, 1)], (INF, 2, 2), INF),
                                      ([(-INF, 0, 1), (-INF, 1, 0)], (1, 2, 2), INF)])
def test_no_width(ctx, orc, p, r, want):
    p, r = np.array(p, dtype=float), np.array(r, dtype=float)
    assert orc.hypervolume(p, r) == want
    assert MO.hypervolume(p, context=ctx).compute(r) == want


@pytest.mark.gpu
@pytest.mark.parametrize("m", [2, 3])
def test_infinite_coordinates(ctx, m):
    for p, r in cases(m, 300):
        assert MO.hypervolume(p, context=ctx).compute(r) == measure(p, r), (p, r)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [2, 3])
def test_infinite_edge_of_a_front(ctx, m):
    # points of no width beside 5000 of some, over several runs and blocks: they add nothing
    rng = np.random.default_rng(m)
    p = np.concatenate([rng.random((5000, m)), rng.random((600, m))])
    p[5000:, 0] = 1.5
    flat = p.copy()
    flat[5000:, 0] = INF
    r = np.full(m, 1.5)
    assert MO.hypervolume(p, context=ctx).compute(r) == pytest.approx(MO.hypervolume(p[:5000], context=ctx).compute(r), rel=1e-13, abs=0)
    r[0] = INF
    assert MO.hypervolume(flat[5000:], context=ctx).compute(r) == 0.0
    assert MO.hypervolume(flat, context=ctx).compute(r) == INF
    flat[5000:, 0] = -INF
    r[0] = 1.5
    assert MO.hypervolume(flat, context=ctx).compute(r) == INF
