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
