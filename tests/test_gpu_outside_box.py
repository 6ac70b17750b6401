"""Positions that their program has not wrapped into the box: the radial distribution and
the differentiable engine must answer as for the wrapped ones."""

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def _unwrapped(N, rho, out, seed=3):
    """A disordered system with a tenth of its coordinates up to `out` boxes outside."""
    x, v, L = ljref.initial_state(N, 1.0, rho, seed)
    rng = np.random.default_rng(N)
    x = np.mod(x[:, :3] + rng.uniform(-0.1, 0.1, (N, 3)), L)
    raw = x + L * rng.integers(-out, out + 1, x.shape) * (rng.random(x.shape) < 0.1)
    near = rng.random(x.shape) < 0.1  # and some just outside a face
    raw = np.where(near & (x < 0.4), x + L, np.where(near & (x > L - 0.4), x - L, raw))
    return raw, raw - np.floor(raw / L) * L, v[:, :3].copy(), L


# half-size cells with the FP32 test, cells with the exact one, all pairs
# (which takes what is less than half a box outside)
@pytest.mark.parametrize("N,rho,bins,rmax,out", [(4000, 0.8, 200, 3.0, 2), (32000, 0.8442, 11000, 3.5, 2),
                                                 (500, 0.8, 100, 4.0, 0)])
def test_rdf_of_unwrapped_positions(N, rho, bins, rmax, out):
    from lennardjonesium import GpuSystem
    raw, x, _, L = _unwrapped(N, rho, out)
    want = ljref.rdf(x, L, bins, rmax)
    with GpuSystem(N, L) as g:
        g.upload(raw)
        got = g.rdf(bins, rmax)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("N", [4000, 23681])  # one launch a pass, separate kernels
def test_adjoint_from_unwrapped_positions(N):
    """Series to 1e-10, gradients to 1e-8 of the largest: rounding of the wrapped start,
    grown over 8 steps."""
    from lennardjonesium import AdjointNVE
    raw, x, v, L = _unwrapped(N, 0.8, 1)
    with AdjointNVE(N, L, 8, checkpoint_every=3) as e:
        pe, p, series = e.forward(raw, v)
        g = e.backward(1.0, 1.0)
        pe0, p0, series0 = e.forward(x, v)
        g0 = e.backward(1.0, 1.0)
    st = ljref.State(x, v)
    st.F, st.pe, st.vir = ljref.forces(x, L)
    want = ljref.run_steps(st, L, 0.005, 8)
    assert np.allclose(series[:, 0], want[:, 2], rtol=1e-10, atol=0)
    assert np.allclose(series, series0, rtol=1e-10, atol=0)
    for k in ("x0", "v0"):
        assert np.abs(g[k] - g0[k]).max() <= 1e-8 * np.abs(g0[k]).max(), k
    for k in ("epsilon", "sigma"):
        assert abs(g[k] - g0[k]) <= 1e-8 * abs(g0[k])
