"""Several host threads, each with a context of its own whose steps take a launch that
fills the GPU, as a pool of simulations runs them: every thread's records and state
must be those of the same system run alone."""

import concurrent.futures as cf

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def _run(args):
    from lennardjonesium import GpuSystem
    N, seed, calls = args
    x, v, L = ljref.initial_state(N, 1.0, 0.8, seed)
    with GpuSystem(N, L) as g:
        g.upload(x, v=v)
        th = np.concatenate([g.step(n) for n in calls])
        return th, g.download()


def test_contexts_on_threads_equal_contexts_alone():
    jobs = [(4000, 1, (7, 50, 1, 30)), (30000, 2, (40, 40)), (30000, 3, (1, 60, 20)), (60000, 4, (25, 25)),
            (500, 5, (200, 1, 99)), (13500, 6, (33, 33, 33))]
    alone = [_run(j) for j in jobs]
    with cf.ThreadPoolExecutor(len(jobs)) as pool:
        for _ in range(3):
            for (th, st), (th0, st0) in zip(pool.map(_run, jobs), alone):
                assert np.array_equal(th, th0)
                for k in ("x", "v", "d", "F"):
                    assert np.array_equal(st[k], st0[k]), k
