"""The three ways a radial distribution histogram is counted -- all pairs, cells with
the exact arithmetic, half-size cells with an FP32 test -- on either side of the
lines between them, bit for bit against the oracle: ragged sizes, thin and dense
systems, a flat box, bins so narrow that FP32 cannot tell them apart, and an
undisturbed lattice, whose distances sit on bin edges by the thousand."""

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu

# N, rho, bins, rmax, jitter
CASES = [
    (130, 0.8, 60, 2.5, 0.3),       # all pairs, one block of atoms
    (2000, 1.0, 100, 4.2, 0.3),     # all pairs, sliced
    (4000, 0.8, 200, 4.0, 0.3),
    (4000, 0.8, 160, 4.0, 0.0),     # the lattice itself
    (4099, 0.3, 333, 4.4, 0.3),
    (30001, 0.05, 77, 2.5, 0.3),
    (32000, 0.8442, 9000, 3.5, 0.3),   # bins of a few error bounds: FP32 test
    (32000, 0.8442, 11000, 3.5, 0.3),  # narrower: exact arithmetic
    (100003, 0.8442, 200, 4.0, 0.3),
]


@pytest.mark.parametrize("N,rho,bins,rmax,jitter", CASES)
def test_histogram_is_the_oracles(N, rho, bins, rmax, jitter):
    from lennardjonesium import GpuSystem
    x, _, L = ljref.initial_state(N, 1.0, rho, 5)
    rng = np.random.default_rng(N + bins)
    x[:, :3] = np.mod(x[:, :3] + rng.uniform(-jitter, jitter, size=(N, 3)), L)
    rmax = min(rmax, L / 2)
    want = ljref.rdf_cells(x, L, bins, rmax) if L >= 3 * rmax else ljref.rdf(x, L, bins, rmax)
    with GpuSystem(N, L) as g:
        g.upload(x)
        got = [g.rdf(bins, rmax) for _ in range(2)]  # the second must not see the first's leftovers
        g.rdf_accumulate(bins, rmax)
        g.rdf_accumulate(bins, rmax)
        total, samples = g.rdf_read()
    assert want.sum() > 0
    assert np.array_equal(got[0], want) and np.array_equal(got[1], want)
    assert samples == 2 and np.array_equal(total, 2 * want)


def test_flat_box():
    from lennardjonesium import GpuSystem
    rng = np.random.default_rng(9)
    box = np.array([60.0, 41.0, 9.5])
    x = rng.uniform(0.0, 1.0, (20011, 3)) * box
    with GpuSystem(20011, box) as g:
        g.upload(x)
        got = g.rdf(150, 3.1)
    assert np.array_equal(got, ljref.rdf(x, box, 150, 3.1))
