"""Contexts that step at the same time on threads of their own share the GPU: those of the
one-launch form take a share of its SMs each, or step as graphs, and neither shows in the
results.  Run one after the other, a launch that fills the GPU each, the same calls take
about as long as without threads; shared, a third to a half (0.75 is asked for)."""

import threading
import time

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def _contexts(sizes, precision="fp64"):
    from lennardjonesium import GpuSystem
    gs = []
    for k, N in enumerate(sizes):
        x, v, L = ljref.initial_state(N, 1.2, 0.8, k + 1)
        g = GpuSystem(N, L, precision=precision)
        g.upload(x, v=v)
        gs.append(g)
    return gs


def _together(gs, calls):
    out, bar = [None] * len(gs), threading.Barrier(len(gs) + 1)

    def run(k):
        bar.wait()
        out[k] = np.concatenate([gs[k].step(n) for n in calls])

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(gs))]
    for t in threads:
        t.start()
    bar.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    return out, time.perf_counter() - t0


# all of them in shares of the SMs; the larger ones as graphs; nearly an atom per thread
@pytest.mark.parametrize("sizes", [(500, 864, 4000, 4096, 6000, 13500), (500, 8192, 8193, 40000, 60000, 189440),
                                   (90000, 500, 500, 4000), (200, 200, 500, 200)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_results_do_not_show_it(sizes, precision):
    calls = (3, 1, 2, 40, 8, 1, 33, 2, 70)
    gs = _contexts(sizes, precision)
    got, _ = _together(gs, calls)
    ends = [g.download() for g in gs]
    for g in gs:
        g.close()
    for k, g in enumerate(_contexts(sizes, precision)):
        want = np.concatenate([g.step(n) for n in calls])
        end = g.download()
        g.close()
        assert np.array_equal(got[k], want), sizes[k]
        for q in ("x", "v", "d", "F"):
            assert np.array_equal(ends[k][q], end[q]), (sizes[k], q)


@pytest.mark.parametrize("N", [500, 4000, 16000])
def test_launches_run_side_by_side(N):
    gs = _contexts([N] * 8)
    ratio = 1.0
    for g in gs:
        g.step(200)
    for _ in range(5):
        t0 = time.perf_counter()
        for g in gs:
            for _ in range(4):
                g.step(200)
        alone = time.perf_counter() - t0
        ratio = min(ratio, _together(gs, (200,) * 4)[1] / alone)
    for g in gs:
        g.close()
    assert ratio < 0.75


def test_async_steps_count_until_they_are_waited_for():
    """Steps that one context has enqueued and not waited for, and another's steps."""
    gs = _contexts((4000, 4000, 30000))
    a, b, c = gs
    a.step_async(500)
    got = b.step(50)
    c.step_async(100)
    a.step_async(20)
    a.synchronize()
    rest = a.step(5), b.step(5), c.step(5)
    for g in gs:
        g.close()
    a, b, c = gs = _contexts((4000, 4000, 30000))
    a.step(520)
    assert np.array_equal(got, b.step(50))
    c.step(100)
    for x, g in zip(rest, gs):
        assert np.array_equal(x, g.step(5))
        g.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_forces_beside_other_contexts(precision):
    """Force evaluations in a share of the SMs and, where the contexts have too many atoms
    together, by the separate kernels: as alone, bit for bit, and no slower than a few
    times that."""
    small, a, large = gs = _contexts((4000, 60000, 90000), precision)
    want = [g.compute_forces() for g in gs]
    F = [g.download()["F"] for g in gs]
    t0 = time.perf_counter()
    for _ in range(20):
        large.compute_forces()
    alone = time.perf_counter() - t0
    for other in ((small,), (a, small)):  # 94 000 atoms together; 154 000
        for g in other:
            g.step_async(2000)
        t0 = time.perf_counter()
        got = [large.compute_forces() for _ in range(20)][-1]
        took = time.perf_counter() - t0
        assert got == want[2]
        assert np.array_equal(large.download()["F"], F[2])
        for g in other:
            g.synchronize()
        assert took < 0.5 + 10 * alone
    for g in gs:
        g.close()


def test_contexts_beside_a_batch():
    """A batch's launches, which take the whole GPU, and contexts of more atoms together than
    it has threads, from threads of their own: all as alone, bit for bit."""
    from test_gpu_batch_active import Batch
    states = [ljref.initial_state(N, 1.2, 0.8, N) for N in (500, 4000, 13500)]
    sizes, calls = (50000, 60000, 4000), (20, 3, 40, 1, 30)
    b, gs = Batch(states), _contexts(sizes)
    rec = []
    t = threading.Thread(target=lambda: rec.extend(b.step(50) for _ in range(8)))
    t.start()
    got, _ = _together(gs, calls)
    t.join()
    for g in gs:
        g.close()
    b.close()
    b, gs = Batch(states), _contexts(sizes)
    assert all(np.array_equal(r, b.step(50)) for r in rec) and len(rec) == 8
    b.close()
    for k, g in enumerate(gs):
        assert np.array_equal(got[k], np.concatenate([g.step(n) for n in calls])), k
        g.close()
