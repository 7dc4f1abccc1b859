"""The own-cell patch by latitude rings against the oracle's RBC_SingInt: the
grids of RBC_Create and the benchmark's, cell counts that leave a block's last
places empty, single and double layer alone and together."""
import math

import numpy as np
import pytest
from scipy.spatial import cKDTree

from rbc3d_gb300 import geometry as G
from rbc3d_gb300.abi import (FP32C, FP32D, FP64, TERM_CORR, TERM_LINEAR, TERM_PME, TERM_REAL, TLIST_RAW, TLIST_RBC,
                              Context)

pytestmark = pytest.mark.gpu
C = 1 / (4 * math.pi)


@pytest.mark.parametrize("nlat,nlon,ncell", [(12, 24, 1), (14, 28, 11), (24, 48, 6), (25, 50, 4), (36, 72, 4)])
def test_ring_patch_matches_oracle(gpu, oracle, nlat, nlon, ncell):
    L = 9.1 if ncell == 1 else 14.0
    rng = np.random.default_rng(nlat)
    cells = G.make_cells(rng, ncell, [L] * 3, 3.2, nlat=nlat, nlon=nlon, with_g=True)
    cells.celltype[:] = np.arange(ncell) % 2
    prm = dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[16] * 3, P=4, nlat=nlat,
               nlon=nlon, ncelltypes=2, viscRat=[5.0, 0.2])
    ctx = []
    for lib in (oracle, gpu):
        c = Context(lib, prm)
        c.set_cells(cells)
        c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
        ctx.append(c)
    # FP64: the separation of the first radial ring (about 0.01) is a difference
    # of positions up to 14, 2e-16 x 14 / 0.01 = 3e-13; the sums differ in order
    # only.  FP32D: interpolated positions to about 2^-47 of 1.4, 1e-14 / 0.005 =
    # 2e-12 a point on the finest grid, and the table position to 2^-47 x 8192 steps
    for c1, c2 in ((C, C), (C, 0.0), (0.0, C)):
        real = TERM_REAL | TERM_CORR | TERM_LINEAR  # the oracle evaluates the three together
        ref, out = (c.matvec(TLIST_RBC, c1, c2, real, FP64) for c in ctx)
        assert np.linalg.norm(out - ref) <= 1e-11 * np.linalg.norm(ref), (c1, c2)
        ref, out = (ctx[1].matvec(TLIST_RBC, c1, c2, TERM_CORR, prec) for prec in (FP64, FP32D))
        assert np.linalg.norm(out - ref) <= 2e-11 * np.linalg.norm(ref), (c1, c2)
    for c in ctx:
        c.close()


def test_shifted_longitudes(gpu, oracle):
    """Longitudes phi(j) = j 2 pi / nlon + 0.3 are not the uniform grid of the
    ring patch and the dense own-cell pass: the general patch, and own-cell
    pairs with mask weights in the cell-list walk."""
    L, ncell = 14.0, 3
    cells = G.make_cells(np.random.default_rng(3), ncell, [L] * 3, 3.2, nlat=12, nlon=24, with_g=True)
    cells.phi = cells.phi + 0.3
    prm = dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[16] * 3, P=4, nlat=12, nlon=24,
               ncelltypes=1, viscRat=[5.0])
    out = []
    for lib in (oracle, gpu):
        c = Context(lib, prm)
        c.set_cells(cells)
        c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
        out.append(c.matvec(TLIST_RBC, C, C, TERM_REAL | TERM_CORR | TERM_LINEAR, FP64))
        if lib is gpu:
            out.append(c.matvec(TLIST_RBC, C, C, TERM_REAL | TERM_CORR | TERM_LINEAR, FP32C))
        c.close()
    ref = np.linalg.norm(out[0])
    assert np.linalg.norm(out[1] - out[0]) <= 1e-11 * ref  # as the uniform grid
    assert np.linalg.norm(out[2] - out[0]) <= 1e-6 * ref   # FP32 pair sums


@pytest.mark.parametrize("n,prec", [(1, FP64), (7, FP64), (33, FP64), (8192, FP64), (8193, FP64), (24000, FP64),
                                    (24001, FP64), (50000, FP64), (50001, FP64), (33, FP32C), (12000, FP32C), (12001, FP32C),
                                    (50001, FP32C), (180001, FP32C)])
def test_few_points(gpu, oracle, n, prec):
    """Velocities at n free points: units of 8 targets with four lanes each
    (of 16 with two above 50000, of 32 above 180000), their remainders, blocks that share a unit (up to 24000 targets in FP64,
    12000 in FP32), and both gathers of the FP64 mesh part (a warp per target
    up to 8192)."""
    L = 14.0
    rng = np.random.default_rng(n)
    cells = G.make_cells(rng, 3, [L] * 3, 3.2, nlat=12, nlon=24, with_g=True)
    prm = dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[16, 18, 20], P=6, nlat=12, nlon=24,
               ncelltypes=1, viscRat=[5.0])
    # at least 0.3 from every surface point: no near-singular item decides on a rounded distance
    x = rng.uniform(0, L, size=(3, 3 * n + 30))
    far = cKDTree(cells.x.T % L, boxsize=L).query(x.T)[0] > 0.3
    x = np.ascontiguousarray(x[:, far][:, :n])
    out = []
    for lib in (oracle, gpu):
        c = Context(lib, prm)
        c.set_cells(cells)
        c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
        c.set_raw_targets(x)
        out.append(c.calc_velocity_field(TLIST_RAW, prec if lib is gpu else FP64))
        c.close()
    # FP64: rounding of the sums; FP32: of single pairs and of the mesh
    tol = 1e-10 if prec == FP64 else 2e-6
    assert x.shape[1] == n and np.linalg.norm(out[1] - out[0]) <= tol * np.linalg.norm(out[0])


@pytest.mark.parametrize("P", [2, 4, 6, 8])
def test_spread_orders(gpu, oracle, P):
    """PME at every even spline order (an odd one's factor vanishes at an even
    mesh's highest wave): the tiled spread's rounds of nodes, full and partly
    filled, all at once or (many rounds) one at a time."""
    L = 14.0
    rng = np.random.default_rng(P)
    cells = G.make_cells(rng, 3, [L] * 3, 3.2, nlat=12, nlon=24, with_g=True)
    prm = dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[24, 20, 18], P=P, nlat=12, nlon=24,
               ncelltypes=1, viscRat=[5.0])
    out = []
    for lib in (oracle, gpu):
        c = Context(lib, prm)
        c.set_cells(cells)
        c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
        out.append(c.matvec(TLIST_RBC, C, C, TERM_PME, FP32C if lib is gpu else FP64))
        c.close()
    # FP32 rounding of the mesh part, as test_few_points
    assert np.linalg.norm(out[1] - out[0]) <= 2e-6 * np.linalg.norm(out[0])
