"""A batch whose systems stop one after another: those left get the GPU of all, and their
records and states stay those they have alone, bit for bit."""

import ctypes
import time

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def P(a):
    return a.ctypes.data_as(ctypes.c_void_p)


class Batch:
    def __init__(self, states):
        from lennardjonesium import _native as nat
        self.lib, self.h, self.states = nat.lib(), ctypes.c_void_p(), states
        table = (nat.BatchSystem * len(states))()
        for q, (x, _, L) in zip(table, states):
            q.particle_count, q.time_delta, q.skin = x.shape[0], 0.005, -1.0
            for k in range(3):
                q.box[k] = L
        nat.check(self.lib.lj_batch_create(table, len(states), 2.5, 0, ctypes.byref(self.h)))
        for s in range(len(states)):
            self.upload(s)

    def upload(self, s):
        x, v, _ = self.states[s]
        assert self.lib.lj_batch_upload_system(self.h, s, P(x), P(v), 4) == 0

    def active(self, s, on):
        assert self.lib.lj_batch_set_active(self.h, s, on) == 0

    def step(self, n):
        rec = np.full((n, len(self.states), 7), -1.0)
        assert self.lib.lj_batch_step(self.h, n, P(rec)) == 0
        return rec

    def close(self):
        self.lib.lj_batch_destroy(self.h)


def test_systems_that_stop_and_start():
    from lennardjonesium import GpuSystem
    sizes = [500, 13500, 864, 4000, 30000]
    states = [ljref.initial_state(N, 1.2, 0.8, N) for N in sizes]
    runs = [(0, 1, 2, 3, 4), (1, 3, 4), (3,), (0, 3), (), (1,), (0, 1, 2, 3, 4)]
    got = [[] for _ in sizes]
    b = Batch(states)
    try:
        for on in runs:
            for s in range(len(sizes)):
                b.active(s, int(s in on))
            rec = b.step(20)
            for s in on:
                got[s].append(rec[:, s])
        b.upload(2)  # an upload starts a system
        b.active(0, 0)
        last = b.step(10)
    finally:
        b.close()
    for s, (x, v, L) in enumerate(states):
        with GpuSystem(sizes[s], L) as g:
            g.upload(x, v=v)
            assert np.array_equal(np.concatenate(got[s]), g.step(20 * len(got[s]))), s
            if s == 2:
                g.upload(x, v=v)
            if s:
                assert np.array_equal(last[:, s], g.step(10)), s


def test_many_systems_in_turns():
    """More systems than blocks (waves), half of them active, then others."""
    x, v, L = ljref.initial_state(500, 1.2, 0.8, 1)
    b = Batch([(x, v, L)] * 1600)
    try:
        for s in range(0, 1600, 2):
            b.active(s, 0)
        a = b.step(12)
        for s in range(1600):
            b.active(s, int(s % 2 == 0 or s > 1500))
        c = b.step(12)
    finally:
        b.close()
    for s in range(3, 1600, 2):
        assert np.array_equal(a[:, s], a[:, 1])
    for s in range(0, 1600, 2):
        assert np.array_equal(c[:, s], a[:, 1])


def test_the_last_system_gets_the_gpu():
    states = [ljref.initial_state(13500, 1.2, 0.8, k) for k in range(40)]
    took = []
    for keep in (40, 1):  # one active of 40; a batch of its own
        b = Batch(states[:keep])
        for s in range(1, keep):
            b.active(s, 0)
        b.step(100)
        best = 1e9
        for _ in range(5):
            t0 = time.perf_counter()
            b.lib.lj_batch_step(b.h, 200, None)
            best = min(best, time.perf_counter() - t0)
        took.append(best)
        b.close()
    assert took[0] < 1.5 * took[1]
