"""A batch's chunk that stops at its iteration bound has stepped all the same: an error
of those steps is reported before the bound."""

import ctypes

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


# 864 atoms step in the cooperative launch, 94 721 in graphs
@pytest.mark.parametrize("N", [864, 94721])
def test_errors_come_before_the_iteration_bound(N):
    from lennardjonesium import _native as nat
    x, v, L = ljref.initial_state(N, 0.722, 0.8442, 5489)
    bad = v.copy()
    bad[5, 1] = np.inf  # a non-finite kinetic energy from the first record on
    table = (nat.BatchSystem * 1)()
    table[0].particle_count, table[0].time_delta, table[0].skin = N, 0.005, -1.0
    for k in range(3):
        table[0].box[k] = L
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib, b = nat.lib(), ctypes.c_void_p()
    nat.check(lib.lj_batch_create(table, 1, 2.5, 0, ctypes.byref(b)))
    try:
        assert lib.lj_batch_set_iteration_limit(b, 3) == 0
        assert lib.lj_batch_upload_system(b, 0, P(x), P(v), 4) == 0
        assert lib.lj_batch_step(b, 64, None) == nat.LJ_ERR_TIMEOUT
        assert b"iteration bound" in lib.lj_batch_last_error(b)
        assert lib.lj_batch_upload_system(b, 0, P(x), P(bad), 4) == 0
        assert lib.lj_batch_step(b, 64, None) == nat.LJ_ERR_NONFINITE
    finally:
        lib.lj_batch_destroy(b)
