"""The 3-objective volume's error against exact integer arithmetic. The terms' own errors are independent and average
out; what is left is the sum's: with one rounding at the volume's size its root mean square over many fronts stays
below 2^-53 of the volume (a tree of additions, several of them rounded at that size, reaches 1.3 2^-53)."""
import bisect

import numpy as np
import pytest

from pagmo2_gb300 import multi_objective as MO

BITS = 60  # coordinates are multiples of 2^-BITS


def exact(p, r):
    """The volume in units of 2^(-3 BITS), by a sweep over z with the staircase of (x, y)."""
    rx, ry, rz = r
    xs, ys, area, total = [], [], 0, 0
    order = sorted(map(tuple, p), key=lambda q: q[2])
    for i, (x, y, z) in enumerate(order):
        at = bisect.bisect_right(xs, x)
        if at == 0 or ys[at - 1] > y:
            if at and xs[at - 1] == x:
                at -= 1
            end = at
            while end < len(xs) and ys[end] >= y:
                end += 1
            left, level = x, ys[at - 1] if at else ry
            for j in range(at, end):
                area += (xs[j] - left) * (level - y)
                left, level = xs[j], ys[j]
            area += ((xs[end] if end < len(xs) else rx) - left) * (level - y)
            xs[at:end], ys[at:end] = [x], [y]
        total += ((order[i + 1][2] if i + 1 < len(order) else rz) - z) * area
    return total


def relative_errors(ctx, n, fronts):
    errors = []
    for seed in range(fronts):
        rng = np.random.default_rng(1000 * n + seed)
        w = rng.random((n, 3)) ** 2
        p = np.round(np.ldexp(w / np.linalg.norm(w, axis=1, keepdims=True), 50)) * 2.0 ** -50
        r = np.full(3, 1.125)
        v = MO.hypervolume(p, context=ctx).compute(r)
        want = exact([[int(c * 2 ** BITS) for c in q] for q in p.tolist()], [int(c * 2 ** BITS) for c in r])
        errors.append((int(v * 2.0 ** 60) * 2 ** (3 * BITS - 60) - want) / want)
    return np.array(errors)


def test_exact_sweep(orc):
    rng = np.random.default_rng(3)
    p = rng.integers(0, 9, (60, 3)) / 8.0
    r = np.full(3, 1.25)
    want = exact([[int(c * 2 ** BITS) for c in q] for q in p.tolist()], [int(c * 2 ** BITS) for c in r])
    assert want / 2 ** (3 * BITS) == pytest.approx(orc.hypervolume(p, r), rel=1e-14)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 300, 2000, 5000])
def test_root_mean_square(ctx, n):
    e = relative_errors(ctx, n, 60)
    assert np.sqrt(np.mean(e * e)) <= 2.0 ** -53, np.sqrt(np.mean(e * e))
