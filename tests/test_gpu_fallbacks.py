"""Forms that small systems no longer take by themselves: the batch's step graphs with
every block size and at their device-side iteration bound, and the differentiable
engine's separate kernels where a candidate row of the one-launch form overflows."""

import ctypes

import numpy as np
import pytest

import ljref
from test_gpu_batch_active import Batch, P

pytestmark = pytest.mark.gpu


# 94 721 atoms step in graphs, and with them every system of the batch
@pytest.mark.parametrize("skin,block", [(0.4, 64), (0.2, 256), (0.3, 128)])
def test_batch_graphs_at_every_block_size(skin, block):
    from lennardjonesium import GpuSystem
    from lennardjonesium import _native as nat
    sizes = [864, 94721, 4000]
    states = [ljref.initial_state(N, 1.2, 0.8, N) for N in sizes]
    table = (nat.BatchSystem * len(sizes))()
    for q, (x, _, L) in zip(table, states):
        q.particle_count, q.time_delta, q.skin = x.shape[0], 0.005, skin
        for k in range(3):
            q.box[k] = L
    lib, b = nat.lib(), ctypes.c_void_p()
    nat.check(lib.lj_batch_create(table, len(sizes), 2.5, 0, ctypes.byref(b)))
    recs = np.zeros((45, len(sizes), 7))
    try:
        assert lib.lj_batch_set_force_block(b, block) == 0
        for s, (x, v, _) in enumerate(states):
            assert lib.lj_batch_upload_system(b, s, P(x), P(v), 4) == 0
        assert lib.lj_batch_step(b, 45, P(recs)) == 0
    finally:
        lib.lj_batch_destroy(b)
    for s, (x, v, L) in enumerate(states):
        with GpuSystem(sizes[s], L, skin=skin, force_block=block) as g:
            g.upload(x, v=v)
            assert np.array_equal(recs[:, s], g.step(45)), s


def test_batch_graphs_stop_at_their_iteration_bound():
    """The device-side loop over 8-step bodies stops after the 3 it may run; the batch steps
    on from a new upload."""
    from lennardjonesium import GpuSystem
    from lennardjonesium import _native as nat
    N = 94721
    x, v, L = ljref.initial_state(N, 1.2, 0.8, 5)
    b = Batch([(x, v, L)])
    try:
        assert b.lib.lj_batch_set_iteration_limit(b.h, 3) == 0
        assert b.lib.lj_batch_step(b.h, 64, None) == nat.LJ_ERR_TIMEOUT
        assert b"(3 iterations)" in b.lib.lj_batch_last_error(b.h)
        assert b.lib.lj_batch_set_iteration_limit(b.h, 0) == 0
        b.upload(0)
        recs = b.step(64)
    finally:
        b.close()
    with GpuSystem(N, L) as g:
        g.upload(x, v=v)
        assert np.array_equal(recs[:, 0], g.step(64))


def test_adjoint_of_more_candidates_than_a_row_holds():
    """A simple cubic lattice of spacing 0.315 sigma with a cutoff of 1.13 sigma: 178 pairs an
    atom, which the exact list's rows of 192 hold, among 388 candidates within the skin,
    which rows of 384 do not.  Forces to 1e-10 of the oracle's sums per atom would need
    its cutoff; instead the energy is summed here, and the gradient held to a central
    difference along a random unit direction (h = 1e-7, relative 1e-4)."""
    from lennardjonesium import AdjointNVE
    n, a, rc, M, dt, h = 14, 0.315, 1.13, 5, 1e-8, 1e-7
    N, L = n ** 3, n * a
    rng = np.random.default_rng(2)
    at = np.arange(n) * a + 0.1
    x = np.stack(np.meshgrid(at, at, at, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-1e-3, 1e-3, (N, 3))
    v = rng.normal(size=(N, 3))
    d = rng.standard_normal(x.shape)
    d /= np.linalg.norm(d)

    def energy(x):
        m6 = rc ** -6
        alpha, beta = -4 * m6 * (m6 - 1), 12 * m6 * (2 * m6 - 1)
        e = 0.0
        for i in range(N - 1):
            r = x[i] - x[i + 1:]
            q = ((r - np.round(r / L) * L) ** 2).sum(1)
            q = q[q < rc * rc]
            e += (4 * q ** -3 * (q ** -3 - 1) + alpha + beta * (q / rc ** 2 - 1)).sum()
        return e

    with AdjointNVE(N, L, M, checkpoint_every=2, time_delta=dt, cutoff_sigma=rc) as e:
        pe, p, series = e.forward(x, v)
        g = e.backward(1.0, 0.0)
        fd = (e.forward(x + h * d, v)[0] - e.forward(x - h * d, v)[0]) / (2 * h)
        again = e.forward(x, v)[2]
    assert np.array_equal(series, again)
    # one free step moves an atom by less than 1e-7: the energy is the start's to 1e-5
    assert abs(series[0, 0] - energy(x)) <= 1e-5 * abs(series[0, 0])
    assert abs((g["x0"] * d).sum() - fd) <= 1e-4 * np.linalg.norm(g["x0"])
