"""What one context or call leaves behind for the next."""
import math

import numpy as np
import pytest

from rbc3d_gb300 import geometry as G
from rbc3d_gb300.abi import Context

pytestmark = pytest.mark.gpu
C = 1 / (4 * math.pi)


def params(L, nlat, nlon):
    return dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[24] * 3, P=6, nlat=nlat, nlon=nlon,
                ncelltypes=1, viscRat=[5.0])


@pytest.mark.parametrize("warp", [0.05, 0.0])
def test_second_grid_on_one_context(gpu, warp):
    """cell_geometry after a change from equispaced longitudes to unequal (or
    shifted) ones is that of a fresh context."""
    L = 14.0
    cells = G.make_cells(np.random.default_rng(1), 2, [L] * 3, 3.2, nlat=12, nlon=24)
    phi = cells.phi + (warp * np.sin(cells.phi) if warp else 0.3)
    geom = []
    for first in (cells.phi, None):
        c = Context(gpu, params(L, 12, 24))
        if first is not None:
            c.set_cell_grid(cells.th, first, cells.w)
            c.cell_geometry(cells.x, 2)
        c.set_cell_grid(cells.th, phi, cells.w)
        geom.append(c.cell_geometry(cells.x, 2))
        c.close()
    for a, b in zip(*geom):
        assert np.array_equal(a, b)  # the same tables, the same kernel

