"""The own-cell patch on rings of more than 256 columns (several columns a
thread, or segments of a ring a block) in every arithmetic, against the oracle, and the FP32M patch on the
grids of test_patch_rings: single and double layer alone and together."""
import math

import numpy as np
import pytest

from rbc3d_gb300 import geometry as G
from rbc3d_gb300.abi import FP32C, FP32D, FP32M, FP64, TERM_CORR, TERM_LINEAR, TERM_REAL, TLIST_RBC, Context

pytestmark = pytest.mark.gpu
C = 1 / (4 * math.pi)
REAL = TERM_REAL | TERM_CORR | TERM_LINEAR  # the oracle evaluates the three together


def contexts(libs, nlat, nlon, ncell):
    L = 9.1 if ncell == 1 else 14.0
    cells = G.make_cells(np.random.default_rng(nlat + nlon), ncell, [L] * 3, 3.2, nlat=nlat, nlon=nlon, with_g=True)
    cells.celltype[:] = np.arange(ncell) % 2
    prm = dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[16] * 3, P=4, nlat=nlat,
               nlon=nlon, ncelltypes=2, viscRat=[5.0, 0.2])
    out = []
    for lib in libs:
        c = Context(lib, prm)
        c.set_cells(cells)
        c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
        out.append(c)
    return out


@pytest.mark.parametrize("nlat,nlon,ncell", [(6, 256, 2), (6, 258, 2), (5, 382, 1), (5, 440, 1), (6, 520, 2), (4, 1400, 1)])
def test_wide_rings(gpu, oracle, nlat, nlon, ncell):
    orc, ctx = contexts((oracle, gpu), nlat, nlon, ncell)
    # bounds as test_patch_rings; FP32C and FP32M: the modes' bound on the velocities
    for c1, c2 in ((C, C), (C, 0.0), (0.0, C)):
        ref = orc.matvec(TLIST_RBC, c1, c2, REAL, FP64)
        out = {p: ctx.matvec(TLIST_RBC, c1, c2, REAL, p) for p in (FP64, FP32C, FP32D, FP32M)}
        norm = np.linalg.norm(ref)
        assert np.linalg.norm(out[FP64] - ref) <= 1e-11 * norm, (c1, c2)
        for p in (FP32C, FP32D, FP32M):
            assert np.linalg.norm(out[p] - ref) <= 1e-6 * norm, (p, c1, c2)
        ref, out = (ctx.matvec(TLIST_RBC, c1, c2, TERM_CORR, p) for p in (FP64, FP32D))
        assert np.linalg.norm(out - ref) <= 2e-11 * np.linalg.norm(ref), (c1, c2)
    orc.close()
    ctx.close()


@pytest.mark.parametrize("nlat,nlon,ncell", [(12, 24, 1), (14, 28, 11), (24, 48, 6), (25, 50, 4), (36, 72, 4)])
def test_fp32m_rings(gpu, nlat, nlon, ncell):
    (ctx,) = contexts((gpu,), nlat, nlon, ncell)
    for c1, c2 in ((C, C), (C, 0.0), (0.0, C)):
        ref, out = (ctx.matvec(TLIST_RBC, c1, c2, REAL, p) for p in (FP64, FP32M))
        assert np.linalg.norm(out - ref) <= 1e-6 * np.linalg.norm(ref), (c1, c2)
    ctx.close()
