"""Index scheme of the FP64 own-cell pair pass (k_pair_own64 in
rbc3d_gb300/csrc/pair.cu), restated on the CPU: one block of OT threads per
(target tile T, source tile S >= T) of a cell's points, thread t taking target
T OT + t and at step s the source (t + s) mod OT; off the diagonal each
evaluation is added to both points.  Tiles of 128, and of 32 where blocks are
few."""
import numpy as np
import pytest


@pytest.mark.parametrize("tile", [32, 128])
@pytest.mark.parametrize("nv", [1, 8, 31, 32, 33, 127, 128, 129, 300, 1250])
def test_every_ordered_pair_once(tile, nv):
    ntile = (nv + tile - 1) // tile
    seen = np.zeros((nv, nv), dtype=np.int64)
    tid = np.arange(tile)
    block = 0
    for T in range(ntile):
        for S in range(T, ntile):
            r, t = block, 0  # the kernel's decoding of the block index
            while r >= ntile - t:
                r -= ntile - t
                t += 1
            assert (t, t + r) == (T, S)
            block += 1
            k = T * tile + tid
            for step in range(tile):
                j = (tid + step) & (tile - 1)
                for w in range(tile // 32):  # a warp's lanes add to distinct sources
                    assert len(set(j[32 * w:32 * (w + 1)].tolist())) == 32
                js = S * tile + j
                ok = (k < nv) & (js < nv)
                np.add.at(seen, (k[ok], js[ok]), 1)
                if S != T:
                    np.add.at(seen, (js[ok], k[ok]), 1)
    assert block == ntile * (ntile + 1) // 2
    assert (seen == 1).all()


@pytest.mark.parametrize("tile", [32, 128])
def test_mask_rows_staged_cover_the_tile(tile):
    """A tile's latitude rings fit in the staged rows of the weight table: at
    most (tile - 1) // nlon + 2 of them."""
    for nlat, nlon in [(25, 50), (12, 24), (64, 128), (6, 8), (3, 200)]:
        nv = nlat * nlon
        cap = min(nlat, (tile - 1) // nlon + 2)
        for T in range((nv + tile - 1) // tile):
            lat0, last = T * tile // nlon, min(nlat - 1, (T * tile + tile - 1) // nlon)
            assert 1 <= last - lat0 + 1 <= cap
            k = np.arange(T * tile, min(nv, T * tile + tile))
            assert ((k // nlon >= lat0) & (k // nlon <= last)).all()
