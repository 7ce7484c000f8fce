"""Threads with contexts of their own that launch the same kernels with different amounts of shared memory at the same
time: a kernel's shared-memory limit is one for all of them, so no call may lower it under another's launch."""
import threading

import numpy as np
import pytest
import torch

from pagmo2_gb300 import _native as N
from pagmo2_gb300 import multi_objective as MO
from pagmo2_gb300 import problems as P
from pagmo2_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def in_threads(works, rounds):
    errors, gate = [], threading.Barrier(len(works))

    def loop(work):
        try:
            with N.Context(0) as ctx:
                want = work(ctx)
                gate.wait()
                for _ in range(rounds):
                    got = work(ctx)
                    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got, want))
        except BaseException as e:  # noqa: BLE001
            errors.append(e)
            gate.abort()

    threads = [threading.Thread(target=loop, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("m", [2, 3, 5])
def test_small_populations(m):
    # device calls one after the other: most of their time is between the limit and the launch
    def work(n):
        p = torch.from_numpy(W.nsga2_points(n, m, layers=5)).cuda()
        out = [torch.zeros(n + 1, dtype=torch.int32, device="cuda") for _ in range(5)]
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()

        def run(ctx):
            for _ in range(50):
                N.check(N.lib().pgx_nsga2_survival_device(ctx.handle, p.data_ptr(), n, m, *(o.data_ptr() for o in out), None,
                                                          stream.cuda_stream))
            stream.synchronize()
            return [o.cpu().numpy() for o in out]

        return run

    in_threads([work(n) for n in (8, 16, 1024, 1000)], 200)


def test_large_populations():
    points = [W.nsga2_points(n, 3, layers=5) for n in (1100, 4500, 9000)]
    in_threads([lambda ctx, p=p: MO.nsga2_survival(p, ctx)[:4] for p in points], 100)


def test_clusters():
    def work(atoms):
        x = W.uniform_batch(N.LENNARD_JONES, atoms, 8, seed=atoms)
        return lambda ctx: P.from_kind(N.LENNARD_JONES, atoms, ctx).batch_gradient(x)

    in_threads([work(a) for a in (200, 400, 1500)], 300)
