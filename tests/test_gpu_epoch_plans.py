"""Several epoch plans at a time: a plan's launches do not depend on the plans made after it (the kernel's
shared-memory limit is one for all of them)."""
import numpy as np
import pytest
import torch

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import archipelago as A
from pagmo2_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def plan(shapes, seed):
    return shapes, [W.uniform_batch(k, p, n, seed=seed + i) for i, (k, p, n, _) in enumerate(shapes)]


@pytest.mark.parametrize("atoms", [120, 170, 300, 1000])
def test_a_smaller_plan_after(ctx, monkeypatch, atoms):
    monkeypatch.setenv("PGX_EPOCH_STAGED", "1")  # the device buffers that launch_device reads are the run's
    # enough clusters for blocks of ten warps, where they fit, beside the rastrigin table
    shapes, batches = plan([(N.LENNARD_JONES, atoms, 5000 if atoms <= 170 else 200, True), (N.RASTRIGIN, 50, 4000, True)], 3)
    small, small_batches = plan([(N.RASTRIGIN, 20, 64, True), (N.ROSENBROCK, 20, 64, True)], 9)
    first = A.Epoch(shapes, ctx)
    want = first.run(batches)
    second = A.Epoch(small, ctx)
    try:
        second.run(small_batches)
        first.launch_device()
        torch.cuda.synchronize()
        again = first.run(batches)
        for (f1, g1), (f2, g2) in zip(want, again):
            assert np.array_equal(f1, f2) and np.array_equal(g1, g2)
    finally:
        second.close()
        first.close()
