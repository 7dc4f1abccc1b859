"""Routes of the pair sums and what hangs on them that the other tests reach
only in part: neighbour lists merged between a target's lanes and a block's
warps, two lanes a target and the mesh part's own accumulator for cell targets,
own-cell pairs of a grid whose weight table does not fit beside the dense pass."""
import math

import numpy as np
import pytest
from scipy.spatial import cKDTree

from rbc3d_gb300 import geometry as G
from rbc3d_gb300.abi import (FP32C, FP32D, FP32M, FP64, TERM_ALL, TERM_CORR, TERM_LINEAR, TERM_REAL, TLIST_RAW,
                             TLIST_RBC, Context)

pytestmark = pytest.mark.gpu
C = 1 / (4 * math.pi)


def context(lib, cells, L, Nb):
    prm = dict(Lb=[L] * 3, alpha=G.alpha_for_cutoff(3.0, 1e-6), rc=3.0, eps=1e-6, Nb=[Nb] * 3, P=4, nlat=cells.nlat,
               nlon=cells.nlon, ncelltypes=1, viscRat=[5.0])
    c = Context(lib, prm)
    c.set_cells(cells)
    c.set_cell_density(f=cells.f, g=cells.g, spl_F=cells.spl_F, spl_G=cells.spl_G)
    return c


@pytest.mark.parametrize("n", [700, 24001, 50001])
def test_points_by_the_surfaces(gpu, oracle, n):
    """Free points 0.03 to 0.4 off a surface, within the near-singular reach of
    0.7, among others beyond it: units shared by a block's warps (FP32: up to
    12000 targets, FP64 24000), four and two lanes a target."""
    L = 14.0
    rng = np.random.default_rng(n)
    cells = G.make_cells(rng, 8, [L] * 3, 3.2, nlat=12, nlon=24, with_g=True)
    nv = 12 * 24
    tree = [cKDTree(cells.x[:, k * nv:(k + 1) * nv].T % L, boxsize=L) for k in range(8)]
    p = rng.integers(0, 8 * nv, size=4000)
    near = cells.x[:, p] + rng.uniform(0.03, 0.4, size=4000) * cells.a3[:, p]
    dist = np.array([t.query(near.T % L)[0] for t in tree])
    dist[p // nv, np.arange(4000)] = np.inf
    near = near[:, dist.min(axis=0) > 1.0][:, :600]  # in reach of its own cell only
    far = rng.uniform(0, L, size=(3, 3 * n + 100))
    dist = np.array([t.query(far.T)[0] for t in tree]).min(axis=0)
    far = far[:, dist > 1.0][:, :n - 600]
    x = np.ascontiguousarray(rng.permutation(np.concatenate([near, far], axis=1), axis=1))
    assert x.shape[1] == n
    out, items = [], []
    for lib, prec in ((oracle, FP64), (gpu, FP64), (gpu, FP32C)):
        c = context(lib, cells, L, 16)
        c.set_raw_targets(x)
        out.append(c.matvec(TLIST_RAW, C, C, TERM_REAL | TERM_CORR | TERM_LINEAR, prec))
        items.append(c.counts()["nearsing_items"])
        c.close()
    assert items[0] >= 600 and items[1] == items[0] and items[2] == items[0]
    norm = np.linalg.norm(out[0])
    # FP64: projections by the constant fit move a correction by its tolerance,
    # 3e-12 of it; FP32: the pair sums' rounding (test_few_points)
    assert np.linalg.norm(out[1] - out[0]) <= 1e-10 * norm
    assert np.linalg.norm(out[2] - out[0]) <= 2e-6 * norm


def test_many_cell_points(gpu, oracle):
    """100,800 cell points: two lanes a target, and in FP32D and FP32M the mesh
    part in an accumulator and on a stream of its own."""
    L = 44.4
    cells = G.make_cells(np.random.default_rng(1), 350, [L] * 3, 2.7, nlat=12, nlon=24, with_g=True)
    out = {}
    for key, lib, prec in (("ref", oracle, FP64), ("fp64", gpu, FP64), ("fp32c", gpu, FP32C), ("fp32d", gpu, FP32D),
                           ("fp32m", gpu, FP32M)):
        c = context(lib, cells, L, 48)
        out[key] = c.matvec(TLIST_RBC, C, C, TERM_ALL, prec)
        c.close()
    norm = np.linalg.norm(out["ref"])
    assert np.linalg.norm(out["fp64"] - out["ref"]) <= 1e-10 * norm
    for key in ("fp32c", "fp32d", "fp32m"):
        assert np.linalg.norm(out[key] - out["ref"]) <= 1e-6 * norm, key


def test_weight_table_too_large_for_the_dense_pass(gpu, oracle):
    """12 x 1720 points: two rows of the FP64 weight table are over 160 KB, and
    own-cell pairs stay in the cell-list walk."""
    L = 9.1
    cells = G.make_cells(np.random.default_rng(1), 1, [L] * 3, 3.2, nlat=12, nlon=1720, with_g=True)
    out = []
    for lib, prec in ((oracle, FP64), (gpu, FP64), (gpu, FP32C)):
        c = context(lib, cells, L, 16)
        out.append(c.matvec(TLIST_RBC, C, C, TERM_REAL | TERM_CORR | TERM_LINEAR, prec))
        c.close()
    norm = np.linalg.norm(out[0])
    # as test_wide_rings
    assert np.linalg.norm(out[1] - out[0]) <= 1e-11 * norm
    assert np.linalg.norm(out[2] - out[0]) <= 1e-6 * norm


@pytest.mark.parametrize("cap", ["0", "7"])
def test_near_stage_capacity_fp64(gpu, monkeypatch, cap):
    """The FP64 near pass past its staged capacity: every item is taken once,
    as test_gpu_parity has it for the FP32 modes."""
    rng = np.random.default_rng(5)
    cells = G.make_cells(rng, 3, [10.0] * 3, 3.2, nlat=12, nlon=24, with_g=True)
    p = rng.integers(0, cells.x.shape[1], size=300)
    x = np.ascontiguousarray(cells.x[:, p] + rng.uniform(0.03, 0.4, size=300) * cells.a3[:, p])
    out = []
    for env in (None, cap):
        if env is not None:
            monkeypatch.setenv("RBC3D_NEAR_STAGE_CAP", env)
        c = context(gpu, cells, 10.0, 16)
        c.set_raw_targets(x)
        v = c.matvec(TLIST_RAW, C, C, TERM_CORR, FP64)
        out.append((v, c.counts()))
        c.close()
    (ref, cref), (v, cnt) = out
    assert cref["nearsing_items"] >= 300
    assert cnt["near_projections"] == cref["near_projections"] and cnt["nearsing_items"] == cref["nearsing_items"]
    assert np.abs(v - ref).max() <= 1e-12 * np.abs(ref).max()
