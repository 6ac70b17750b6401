"""The differentiable engine's one-launch passes (up to 23 680 atoms) at the sizes where
the lanes per atom change, at the last size of this form and the first beyond it,
in a box whose candidate list has no room for a skin, and in a thin system whose
cells are scanned over all blocks.  The trajectory is held to the oracle's (1e-10, the
bound of the engine's own test) and the gradient to a central difference along a
random unit direction (h = 1e-6, 1e-4 relative, as there)."""

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu

DT, H = 0.005, 1e-6


@pytest.mark.parametrize("N,rho,steps,every", [
    (500, 1.13, 12, 5),       # 3 cells of edge 2.54: no skin
    (5920, 0.8, 8, 3), (5921, 0.8, 8, 8),
    (11840, 0.8, 8, 3), (11841, 0.8, 8, 1),
    (12000, 0.06, 8, 3),      # more than 1024 cells
    (23680, 0.8, 6, 4), (23681, 0.8, 6, 4),
])
def test_one_launch_passes(N, rho, steps, every):
    from lennardjonesium import AdjointNVE
    x, v, L = ljref.initial_state(N, 1.2, rho, N)
    rng = np.random.default_rng(N)
    x, v = x[:, :3].copy(), v[:, :3].copy()
    x = np.mod(x + rng.uniform(-0.05, 0.05, x.shape), L)
    st = ljref.State(x, v)
    st.F, st.pe, st.vir = ljref.forces(x, L)
    want = ljref.run_steps(st, L, DT, steps)
    dx = rng.standard_normal(x.shape)
    dx /= np.linalg.norm(dx)
    with AdjointNVE(N, L, steps, checkpoint_every=every, time_delta=DT) as e:
        pe, p, series = e.forward(x, v)
        g = e.backward(1.0, 1.0)
        fd = (sum(e.forward(x + H * dx, v)[:2]) - sum(e.forward(x - H * dx, v)[:2])) / (2 * H)
    assert np.allclose(series[:, 0], want[:, 2], rtol=1e-10, atol=0)
    assert np.allclose(series[:, 1], want[:, 4], rtol=1e-10, atol=0)
    assert np.allclose(series[:, 2], want[:, 1], rtol=1e-10, atol=0)
    ad = float((g["x0"] * dx).sum())
    assert abs(ad - fd) <= 1e-4 * abs(fd)
