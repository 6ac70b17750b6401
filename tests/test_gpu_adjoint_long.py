"""A one-launch pass so long that the barrier's votes are cleared on the way (after some
hundred rebuilds): every sum depends on the state alone, so a pass of many steps must
agree bit for bit with the shorter one from the same start, and its energy with the
conserved one."""

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def test_votes_of_a_long_pass():
    from lennardjonesium import AdjointNVE
    N = 4000
    x, v, L = ljref.initial_state(N, 1.5, 0.8, 11)
    x, v = x[:, :3].copy(), v[:, :3].copy()
    with AdjointNVE(N, L, 300, checkpoint_every=300) as e:
        short = e.forward(x, v)[2]
    with AdjointNVE(N, L, 6000, checkpoint_every=3000) as e:
        long = e.forward(x, v)[2]
        again = e.forward(x, v)[2]
    assert np.array_equal(long[:300], short)
    assert np.array_equal(long, again)
    energy = long[:, 0] + long[:, 2]
    # a list that missed its rebuilds loses pairs of a few times 0.1 each
    assert np.abs(energy - energy[0]).max() <= 1e-3 * abs(energy[0])
