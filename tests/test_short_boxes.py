"""Cells that nearly meet their own image: boxes shorter than a cell's extent
plus the cutoff, which rbc3d_create accepts (rc <= L / 3).  The own-cell pass
takes a cell's pairs relative to its first point; where a pair's minimum image
is another one, the cell-list walk takes the cell's pairs."""
import math

import numpy as np
import pytest

from rbc3d_gb300 import geometry as G
from rbc3d_gb300.abi import (FP32C, FP32D, FP64, TERM_CORR, TERM_LINEAR, TERM_REAL, TLIST_RBC, Context)

pytestmark = pytest.mark.gpu
C = 1 / (4 * math.pi)


@pytest.mark.parametrize("L,centres", [([3.9] * 3, [[1.0, 2.0, 1.5]]), ([4.1] * 3, [[4.0, 0.1, 2.0]]),
                                       ([3.9, 9.1, 9.1], [[0.3, 2.0, 2.0], [2.0, 6.0, 6.0]]),
                                       ([4.5] * 3, [[1.0, 2.0, 1.5]])])
def test_own_image_pairs(gpu, oracle, L, centres):
    rc = min(L) / 3.001
    rng = np.random.default_rng(7)
    cells = G.make_cells(rng, len(centres), L, 1.0, with_g=True, centres=np.array(centres),
                         rotations=[np.eye(3)] * len(centres))
    prm = dict(Lb=L, alpha=G.alpha_for_cutoff(rc, 1e-6), rc=rc, eps=1e-6, Nb=[16] * 3, P=4, nlat=25, nlon=50,
               ncelltypes=1, viscRat=[5.0])
    real = TERM_REAL | TERM_CORR | TERM_LINEAR
    out, pairs = {}, {}
    for key, lib, prec in (("oracle", oracle, FP64), ("fp64", gpu, FP64), ("fp32c", gpu, FP32C), ("fp32d", gpu, FP32D)):
        c = Context(lib, prm)
        c.set_cells(cells)
        c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
        out[key] = c.matvec(TLIST_RBC, C, C, real, prec)
        pairs[key] = c.counts()["pairs_within_rc"]
        c.close()
    ref = np.linalg.norm(out["oracle"])
    # every pair within rc once: FP64 decides as the oracle, but for pairs at the cutoff to rounding
    assert abs(pairs["fp64"] - pairs["oracle"]) <= 2
    # FP64: the sums' order and the patch's rounding (as test_patch_rings); FP32:
    # the pair sums' bound
    assert np.linalg.norm(out["fp64"] - out["oracle"]) <= 1e-11 * ref
    for key in ("fp32c", "fp32d"):
        assert np.linalg.norm(out[key] - out["oracle"]) <= 1e-6 * ref, key
