"""What one context or call leaves behind for the next."""
import math
import threading

import numpy as np
import pytest

from rbc3d_gb300 import geometry as G
from rbc3d_gb300.abi import FP32C, FP32D, FP32M, FP64, TERM_ALL, TLIST_RBC, TLIST_WALL, Context, RBC3DError

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



def test_larger_grid_after_a_smaller_one(gpu):
    """The shared-memory limit of a kernel is the process's: a context of a
    smaller grid leaves it where a larger one needs it."""
    L = 14.0
    ctx, geom = [], []
    for nlat, nlon in ((36, 72), (33, 66)):
        cells = G.make_cells(np.random.default_rng(2), 1, [L] * 3, 3.2, nlat=nlat, nlon=nlon)
        c = Context(gpu, params(L, nlat, nlon))
        c.set_cell_grid(cells.th, cells.phi, cells.w)
        geom.append(c.cell_geometry(cells.x, 1))
        ctx.append((c, cells))
    c, cells = ctx[0]
    for a, b in zip(c.cell_geometry(cells.x, 1), geom[0]):
        assert np.array_equal(a, b)
    for c, _ in ctx:
        c.close()


def test_grids_in_two_threads(gpu):
    """A context per host thread, each of another grid, whose kernels take
    other amounts of shared memory: every call of both succeeds."""
    L, failed = 14.0, []

    def work(nlat, nlon):
        try:
            cells = G.make_cells(np.random.default_rng(nlat), 2, [L] * 3, 3.2, nlat=nlat, nlon=nlon, with_g=True)
            c = Context(gpu, params(L, nlat, nlon))
            c.set_cells(cells)
            c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
            ref = {p: c.matvec(TLIST_RBC, C, C, TERM_ALL, p) for p in (FP64, FP32D, FP32M)}
            for _ in range(40):
                for p, r in ref.items():
                    v = c.matvec(TLIST_RBC, C, C, TERM_ALL, p)
                    # the atomics' order: of FP64 sums, and of FP32 mesh sums (test_few_points)
                    assert np.linalg.norm(v - r) <= (1e-13 if p == FP64 else 2e-6) * np.linalg.norm(r)
            c.close()
        except Exception as e:
            failed.append((nlat, e))

    threads = [threading.Thread(target=work, args=g) for g in ((12, 24), (25, 50))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("prec", [FP64, FP32C])
def test_cells_replaced_after_a_failed_matvec(gpu, prec):
    """A wall-list matvec before prepare_sing_int_on_wall is refused with the
    mesh part already under way; cells and densities replaced right after it
    give a fresh context's velocities."""
    L = 14.0
    wall = G.make_tube(5.0, L, 16, 8, (7.0, 7.0))
    rng = np.random.default_rng(4)
    first, second = (G.make_cells(rng, n, [L] * 3, 2.8, with_g=True) for n in (12, 3))
    fw = rng.normal(size=(3, wall.nvert))
    out = []
    for fails in (20, 0):
        c = Context(gpu, params(L, 25, 50))
        for k in range(max(fails, 1)):
            if fails:
                c.set_cells(first)
                c.set_cell_density(f=first.f, g=first.g, spl_F=first.spl_F, spl_G=first.spl_G)
            c.set_walls(wall)
            c.set_wall_density(fw)
            if fails:
                with pytest.raises(RBC3DError) as e:
                    c.matvec(TLIST_WALL, C, C, TERM_ALL, prec)
                assert e.value.code == 6  # ERR_STATE
            c.set_cells(second)
            c.set_cell_density(f=second.f, g=second.g, spl_F=second.spl_F, spl_G=second.spl_G)
            v = c.matvec(TLIST_RBC, C, C, TERM_ALL, prec)
            out.append(v)
        c.close()
    for v in out[:-1]:
        # the atomics' order, as test_grids_in_two_threads
        assert np.linalg.norm(v - out[-1]) <= (1e-13 if prec == FP64 else 2e-6) * np.linalg.norm(out[-1])
