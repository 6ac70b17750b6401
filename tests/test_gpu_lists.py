"""Both forms of the neighbour-list build -- a warp per list cell, an atom per lane --
on either side of the line between them (12 atoms per cell), at sizes that leave
ragged cells, runs off the 16-byte boundary and columns that wrap, in a cubic and a
flat box: the pair set the force kernel uses must be the oracle's, pair by pair and
bit by bit in r^2."""

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu


def _gas(N, box, rng):
    """N points no two of which are closer than 0.86 (a jittered lattice with holes)."""
    n = np.ones(3, dtype=int)
    while n.prod() < N:
        n[np.argmax(box / n)] += 1
    a = box / n
    sites = rng.permutation(n.prod())[:N]
    g = np.stack(np.unravel_index(sites, n), axis=1)
    room = np.maximum(0.5 * (a - 0.86), 0.0)
    return np.mod((g + 0.5) * a + rng.uniform(-1.0, 1.0, (N, 3)) * np.minimum(room, 0.4), box)


@pytest.mark.parametrize("N,rho,shape,precision", [
    (70001, 0.05, (1, 1, 1), "fp64"),    # thin: an atom per lane
    (70001, 0.48, (1, 1, 1), "fp64"),    # just below the line
    (70001, 0.56, (1, 1, 1), "fp64"),    # just above: a warp per cell
    (66003, 0.9, (3, 3, 1), "fp64"),     # flat box
    (66003, 0.3, (1, 4, 4), "fp64"),
    (66003, 0.9, (3, 3, 1), "mixed"),
    (4099, 0.2, (1, 1, 1), "mixed"),
])
def test_lists_hold_the_oracles_pairs(N, rho, shape, precision):
    from lennardjonesium import GpuSystem
    rng = np.random.default_rng(N)
    box = np.array(shape, dtype=float)
    box *= (N / rho / box.prod()) ** (1 / 3)
    x = _gas(N, box, rng)
    oi, oj, _, o2 = ljref.pairs(x, box, 2.5)
    oi, oj = np.minimum(oi, oj), np.maximum(oi, oj)
    with GpuSystem(N, box, precision=precision) as g:
        g.upload(x)
        gi, gj, _, g2 = g.debug_pairs()
        st = g.stats()
    assert len(gi) == len(oi) > 0
    a, b = np.lexsort((gj, gi)), np.lexsort((oj, oi))
    assert np.array_equal(gi[a], oi[b]) and np.array_equal(gj[a], oj[b])
    assert np.array_equal(g2[a].view(np.uint64), o2[b].view(np.uint64))
    assert 0 < st["max_neighbors"] <= st["neighbor_capacity"]
