"""Batches whose systems have somewhat more atoms than their blocks have threads, where two
lanes share a row, on either side of the line: records and states as alone, bit for bit."""

import numpy as np
import pytest

import ljref
from test_gpu_batch_active import Batch, P

pytestmark = pytest.mark.gpu


# 740 blocks of 128 threads: 1.27, 1.06, 1.5 and 1.51 atoms a thread
@pytest.mark.parametrize("sizes", [(60000, 60000), (50000, 50001), (71040, 71040), (71500, 71500), (120000,)])
def test_batch_equals_alone(sizes):
    from lennardjonesium import GpuSystem
    states = [ljref.initial_state(N, 1.2, 0.8, N + k) for k, N in enumerate(sizes)]
    b = Batch(states)
    try:
        rec = b.step(30)
        end = [np.zeros((N, 4)) for N in sizes]
        for s, a in enumerate(end):
            assert b.lib.lj_batch_download_system(b.h, s, P(a), None, None, 4) == 0
    finally:
        b.close()
    for s, (x, v, L) in enumerate(states):
        with GpuSystem(sizes[s], L) as g:
            g.upload(x, v=v)
            assert np.array_equal(rec[:, s], g.step(30)), s
            assert np.array_equal(end[s][:, :3], g.download()["x"][:, :3]), s
