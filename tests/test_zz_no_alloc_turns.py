"""lj_gpu_rdf_noalloc with one array for all calls (collected after test_zz_no_alloc.py)."""

import numpy as np
import pytest

import ljref
from test_zz_no_alloc import _noalloc, _positions

pytestmark = pytest.mark.gpu


def test_rdf_noalloc_calls_of_different_grids_in_turn():
    """All calls share one array: histograms of systems with many cells and few, of each
    form in turn, are the oracle's whatever the call before left there."""
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    systems = []
    for N, rho, nbins, rmax in ((32000, 0.05, 50, 2.0), (4000, 0.8, 200, 4.0), (864, 0.8442, 200, 4.0),
                                (32000, 0.8442, 11000, 3.5), (130000, 0.8442, 100, 2.5)):
        x, box = _positions(N, rho, 9)
        rmax = min(rmax, box / 2)
        want = ljref.rdf_cells(x, box, nbins, rmax) if box >= 3 * rmax else ljref.rdf(x, box, nbins, rmax)
        systems.append((x, box, nbins, rmax, want))
    for k in (0, 1, 4, 2, 3, 0, 4, 1, 3, 3, 2, 0):
        x, box, nbins, rmax, want = systems[k]
        rc, got = _noalloc(x, box, nbins, rmax, stream)
        assert rc == 0 and np.array_equal(got, want), k
