"""Step graphs of the sizes that only they step (all others' steps are one launch when
they step alone): calls of every length, so that each graph is built and launched, must
equal steps run one kernel per phase bit for bit; and a short first call must not wait
for graphs that it does not use."""

import time

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,rho", [(100003, 0.8442), (100003, 0.2), (200000, 0.8442)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_graphs_equal_one_kernel_per_phase(N, rho, precision):
    from lennardjonesium import GpuSystem
    x, v, L = ljref.initial_state(N, 1.5, rho, 7)
    with GpuSystem(N, L, precision=precision) as a, GpuSystem(N, L, precision=precision) as b:
        for g in (a, b):
            g.upload(x, v=v)
        # direct launches; the 8-step graph; both lengths; the long one from a short call on
        calls = [3, 11, 40, 130, 45, 32]
        th = [a.step(n) for n in calls]
        for n, got in zip(calls, th):
            b.step_timed(n - 1)
            assert np.array_equal(got[-1], b.step(1)[-1]), n
        sa, sb = a.download(), b.download()
        assert a.stats()["list_builds"] == b.stats()["list_builds"]
        assert a.stats()["steps"] == b.stats()["steps"] == sum(calls)
    for k in ("x", "v", "d", "F"):
        assert np.array_equal(sa[k], sb[k]), k
    assert np.array_equal(np.concatenate(th)[:, 0], np.cumsum(np.full(sum(calls), 0.005)))


def test_first_step_builds_no_graph():
    """A first step is one to two tenths of a millisecond of launches; with the graphs
    built in it, it took five."""
    from lennardjonesium import GpuSystem
    x, v, L = ljref.initial_state(200000, 1.5, 0.8, 7)
    took = []
    for _ in range(4):
        with GpuSystem(200000, L) as g:
            g.upload(x, v=v)
            t0 = time.perf_counter()
            g.step(1)
            took.append(time.perf_counter() - t0)
    assert min(took) < 2e-3
