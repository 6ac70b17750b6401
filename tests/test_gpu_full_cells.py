"""The list form of an atom per lane in cells of more than 32 atoms: such systems build
their lists so in a batch whose other system is too large for the one-launch form, and
by a warp per atom when they step alone."""

import ctypes

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,rho", [(864, 0.8442), (1000, 0.8442), (1200, 1.0)])  # 32, 37, 44 atoms a cell
def test_batch_equals_alone(N, rho):
    from lennardjonesium import GpuSystem
    from lennardjonesium import _native as nat
    states = [ljref.initial_state(N, 1.3, rho, 5), ljref.initial_state(94721, 1.0, 0.3, 6)]
    table = (nat.BatchSystem * 2)()
    for q, (x, _, L) in zip(table, states):
        q.particle_count, q.time_delta, q.skin = x.shape[0], 0.005, -1.0
        for k in range(3):
            q.box[k] = L
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib, b = nat.lib(), ctypes.c_void_p()
    nat.check(lib.lj_batch_create(table, 2, 2.5, 0, ctypes.byref(b)))
    recs = np.zeros((40, 2, 7))
    F = np.zeros((N, 4))
    try:
        for s, (x, v, _) in enumerate(states):
            assert lib.lj_batch_upload_system(b, s, P(x), P(v), 4) == 0
        assert lib.lj_batch_step(b, 40, P(recs)) == 0
        assert lib.lj_batch_download_system(b, 0, None, None, P(F), 4) == 0
    finally:
        lib.lj_batch_destroy(b)
    x, v, L = states[0]
    with GpuSystem(N, L) as g:
        g.upload(x, v=v)
        want = g.step(40)
        end = g.download()
    assert np.array_equal(recs[:, 0], want)
    assert np.array_equal(F[:, :3], end["F"][:, :3])
    F0, _, _ = ljref.forces(end["x"][:, :3], L, 2.5)
    S = ljref.force_abs_sum(end["x"][:, :3], L, 2.5)
    assert np.all(np.abs(F[:, :3] - F0[:, :3]) <= 1e-12 * S[:, None])
