"""Systems that step in one cooperative launch (LJ force; up to 94 720 atoms, and 113 665
to 189 440).

The launch's pair rows are shared by 16, 8, 4, 2 or 1 lanes per atom, its lists
are built by a warp per atom or a thread per atom, and its cells are scanned in
shared memory or over all blocks: each by a rule on the system's size.  The sums
are defined so that none of this can be seen, so steps must equal, bit for bit,
steps run one kernel per phase (lj_gpu_step_timed), at the sizes on either side
of every line.
"""

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu

# 740 blocks of 128 threads: 16 lanes up to 5920 atoms, 8 to 11840, 4 to 23680, 2 to
# 47360, 1 to 94720; above 113664 a thread takes two atoms, 189440 is the largest system.
# Up to 4096 atoms (and 1024 cells) every block sorts all.  rho 0.05 has more than 4096 list
# cells and about one atom in each; 40 and 200 atoms are boxes under 3 cells.
CASES = [(1, 0.001), (9, 0.01), (40, 0.8), (200, 0.8), (500, 0.8), (513, 1.0), (1024, 0.8), (1025, 0.02),
         (4096, 0.8), (4097, 0.8), (5920, 0.8442), (5921, 0.8442),
         (11841, 0.7), (23681, 0.8442), (30000, 0.05), (30000, 0.3), (47361, 0.8442), (80001, 0.05), (94720, 0.8442), (94721, 0.8442),
         (113665, 0.8442), (150000, 0.3), (189440, 0.8442), (189441, 0.8442)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N,rho", CASES)
def test_steps_equal_one_kernel_per_phase(N, rho, precision):
    from lennardjonesium import GpuSystem
    x, v, L = ljref.initial_state(N, 1.5, rho, N) if N > 9 else (None, None, 10.0)
    if x is None:
        rng = np.random.default_rng(N)
        x, v = 3.0 * np.arange(N)[:, None] * [1, 0, 0] % 9.0 + rng.uniform(0.0, 0.9, (N, 3)), rng.normal(size=(N, 3))
        x[:, 1] += 3.0 * (np.arange(N) // 3)
    with GpuSystem(N, L, precision=precision) as a, GpuSystem(N, L, precision=precision) as b:
        for g in (a, b):
            g.upload(x, v=v)
        one = a.step(25)
        b.step_timed(24)
        two = b.step(1)
        sa, sb = a.download(), b.download()
        assert a.stats()["list_builds"] == b.stats()["list_builds"] >= 1
    assert np.array_equal(one[-1], two[-1])
    for k in ("x", "v", "d", "F"):
        assert np.array_equal(sa[k], sb[k]), k


@pytest.mark.parametrize("N,rho", [(200, 0.8), (500, 0.8), (5921, 0.8442), (30000, 0.05), (47361, 0.8442)])
def test_forces_match_the_oracle(N, rho):
    """One force evaluation (its own mode of the launch): 1e-12 of each atom's sum of
    |pair forces|, the bound of the parity tests."""
    from lennardjonesium import GpuSystem
    x, _, L = ljref.initial_state(N, 1.0, rho, 3)
    x = np.array(x[:, :3])
    x = np.mod(x + np.random.default_rng(N).uniform(-0.08, 0.08, x.shape), L)
    F0, pe0, w0 = ljref.forces(x, L, 2.5)
    S = ljref.force_abs_sum(x, L, 2.5)
    with GpuSystem(N, L) as g:
        g.upload(x)
        pe, w = g.compute_forces()
        F = g.download()["F"]
    assert np.all(np.abs(F[:, :3] - F0[:, :3]) <= 1e-12 * S[:, None])
    assert abs(pe - pe0) <= 1e-12 * abs(pe0) and abs(w - w0) <= 1e-12 * max(abs(w0), S.sum())


@pytest.mark.parametrize("sizes", [(500, 5921, 94721), (94720, 113664, 40000), (113665, 864, 150000), (189441, 189440)])
def test_batch_of_both_forms_equals_single_systems(sizes):
    """A batch with a system that steps in graphs takes all of them through graphs; with
    none, all in one launch: each system's records and state as it has alone."""
    import ctypes
    from lennardjonesium import GpuSystem
    from lennardjonesium import _native as nat
    states = [ljref.initial_state(N, 1.2, 0.8442, N) for N in sizes]
    table = (nat.BatchSystem * len(sizes))()
    for q, (x, _, L) in zip(table, states):
        q.particle_count, q.time_delta, q.skin = x.shape[0], 0.005, -1.0
        for k in range(3):
            q.box[k] = L
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib, b = nat.lib(), ctypes.c_void_p()
    nat.check(lib.lj_batch_create(table, len(sizes), 2.5, 0, ctypes.byref(b)))
    recs = np.zeros((20, len(sizes), 7))
    try:
        for s, (x, v, _) in enumerate(states):
            nat.check(lib.lj_batch_upload_system(b, s, P(x), P(v), 4))
        assert lib.lj_batch_step(b, 20, P(recs)) == 0
        got = [[np.zeros_like(x) for _ in range(3)] for x, _, _ in states]
        for s, (x, v, F) in enumerate(got):
            nat.check(lib.lj_batch_download_system(b, s, P(x), P(v), P(F), 4))
    finally:
        lib.lj_batch_destroy(b)
    for s, (x, v, L) in enumerate(states):
        with GpuSystem(x.shape[0], L) as g:
            g.upload(x, v=v)
            ref = g.step(20)
            st = g.download()
        assert np.array_equal(recs[:, s], ref), s
        for k, a in zip("xvF", got[s]):
            assert np.array_equal(a[:, :3], st[k][:, :3]), (s, k)
