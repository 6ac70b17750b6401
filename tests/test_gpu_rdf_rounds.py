"""Histograms of systems so large that a block counts many rounds of atoms: the simple cubic
lattice, of which every atom has 6 neighbours at distance 1 and 12 at sqrt 2.  Bins lie
so that both distances are well inside theirs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one round of atoms, two, and seven of which five fit the 32-bit counts of a block
@pytest.mark.parametrize("side", [40, 80, 144])
def test_lattice(side):
    from lennardjonesium import GpuSystem
    N = side ** 3
    at = np.arange(side) + 0.25
    x = np.stack(np.meshgrid(at, at, at, indexing="ij"), axis=-1).reshape(-1, 3)
    x = x[np.random.default_rng(side).permutation(N)]
    want = np.zeros(5, dtype=np.uint64)
    want[3], want[4] = 6 * N, 12 * N
    with GpuSystem(N, float(side)) as g:
        g.upload(x)
        once = g.rdf(5, 1.5)
        for _ in range(3):
            g.rdf_accumulate(5, 1.5)
        total, samples = g.rdf_read()
    assert np.array_equal(once, want)
    assert samples == 3 and np.array_equal(total, 3 * want)
