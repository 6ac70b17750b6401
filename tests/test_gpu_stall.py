"""A wait between the blocks of a cooperative launch that runs out (a launch without one of
its blocks, whose arrival the others wait for in vain, about a second).  The call must
return LJ_ERR_TIMEOUT, so must every later one until the state is uploaded again, and
from then on results are those of a fresh context."""

import ctypes

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def P(a):
    return a.ctypes.data_as(ctypes.c_void_p)


# sorted by every block for itself, cells scanned by each block, and over all of them
@pytest.mark.parametrize("N,rho", [(4000, 0.8), (30000, 0.8), (60000, 0.05)])
@pytest.mark.parametrize("call", ["step", "async"])
def test_context(N, rho, call):
    from lennardjonesium import GpuSystem
    from lennardjonesium import _native as nat
    x, v, L = ljref.initial_state(N, 1.2, rho, N)
    with GpuSystem(N, L) as g:
        g.upload(x, v=v)
        want = g.step(40)
        state = g.download()
    with GpuSystem(N, L) as g:
        lib, h = nat.lib(), g._ctx
        g.upload(x, v=v)
        g.step(3)
        assert lib.lj_gpu_debug_stall(h) == 0
        if call == "step":
            assert lib.lj_gpu_step(h, 1000, None) == nat.LJ_ERR_TIMEOUT
        else:  # the launch that ran out is not the last one
            assert lib.lj_gpu_step_async(h, 1000) == 0
            assert lib.lj_gpu_step_async(h, 10) == 0
            assert lib.lj_gpu_synchronize(h) == nat.LJ_ERR_TIMEOUT
        pe = ctypes.c_double()
        for _ in range(3):
            assert lib.lj_gpu_step(h, 5, None) == nat.LJ_ERR_TIMEOUT
            assert lib.lj_gpu_compute_forces(h, ctypes.byref(pe), None) == nat.LJ_ERR_TIMEOUT
        assert lib.lj_gpu_step_timed(h, 2, ctypes.byref(nat.PhaseTimes())) == nat.LJ_ERR_TIMEOUT
        assert lib.lj_gpu_debug_pairs(h, 0, None, None, None, None) == -nat.LJ_ERR_TIMEOUT
        g.upload(x, v=v)
        got = g.step(40)
        again = g.download()
        # the device's step count places these records
        g.step_timed(4)
        a = g.step(1)
    assert np.array_equal(got, want)
    for k in ("x", "v", "d", "F"):
        assert np.array_equal(again[k], state[k]), k
    assert np.isfinite(a).all() and a[0, 0] == pytest.approx(45 * 0.005, rel=1e-12)


def test_batch():
    from lennardjonesium import _native as nat
    sizes = [864, 30000, 4000]
    states = [ljref.initial_state(N, 1.2, 0.8, N) for N in sizes]
    table = (nat.BatchSystem * len(sizes))()
    for q, (x, _, L) in zip(table, states):
        q.particle_count, q.time_delta, q.skin = x.shape[0], 0.005, -1.0
        for k in range(3):
            q.box[k] = L
    lib, b = nat.lib(), ctypes.c_void_p()
    nat.check(lib.lj_batch_create(table, len(sizes), 2.5, 0, ctypes.byref(b)))

    def upload(s):
        assert lib.lj_batch_upload_system(b, s, P(states[s][0]), P(states[s][1]), 4) == 0

    try:
        for s in range(3):
            upload(s)
        want, got = np.zeros((40, 3, 7)), np.zeros((40, 3, 7))
        assert lib.lj_batch_step(b, 40, P(want)) == 0
        assert lib.lj_batch_debug_stall(b) == 0
        assert lib.lj_batch_step(b, 1000, None) == nat.LJ_ERR_TIMEOUT
        for s in (1, 0):
            assert lib.lj_batch_step(b, 5, None) == nat.LJ_ERR_TIMEOUT
            upload(s)
        assert lib.lj_batch_step(b, 5, None) == nat.LJ_ERR_TIMEOUT
        upload(2)
        assert lib.lj_batch_step(b, 40, P(got)) == 0
    finally:
        lib.lj_batch_destroy(b)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("N", [4000, 23680])
def test_adjoint(N):
    from lennardjonesium import AdjointNVE
    from lennardjonesium import _native as nat
    x, v, L = ljref.initial_state(N, 1.2, 0.8, N)
    x, v = x[:, :3].copy(), v[:, :3].copy()
    with AdjointNVE(N, L, 30, checkpoint_every=7) as e:
        lib, h = nat.lib(), e._ctx
        want = e.forward(x, v)
        grad = e.backward(1.0, 1.0)
        out = np.zeros(2)
        assert lib.lj_adj_debug_stall(h) == 0
        assert lib.lj_adj_forward(h, P(x), P(v), 3, P(out), None) == nat.LJ_ERR_TIMEOUT
        got = e.forward(x, v)
        assert lib.lj_adj_debug_stall(h) == 0
        assert lib.lj_adj_backward(h, 1.0, 1.0, None, None, 3, None, None) == nat.LJ_ERR_TIMEOUT
        again = e.backward(1.0, 1.0)
    assert got[:2] == want[:2] and np.array_equal(got[2], want[2])
    for k in grad:
        assert np.array_equal(again[k], grad[k]), k
