"""The tensor-core screen at the edges of its tiles: column counts around the
padding steps, neighbour rows that begin and end inside a group of 8 slots,
dense and hashed grids, items split into slices, points beyond every bound.
The lists must be the oracle's exactly (integers, no tolerance)."""
import numpy as np
import pytest

from tests.test_gpu_parity import assert_same, tile_points

pytestmark = pytest.mark.gpu


# n + 4 columns pad to 32 at n = 28 and to 48 at n = 29, to 96 at 92, 112 at 93,
# 128 at 124 and 144 at 125
@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("n,k,N", [(16, 1, 2003), (28, 2, 5001), (29, 6, 9003), (92, 3, 4099), (93, 6, 4097),
                                   (124, 6, 3007), (125, 6, 3001)])
def test_screen_tile_edges(oracle, n, k, N, stamp):
    pts = tile_points(n, N, 3.0, 500 + n)
    st = assert_same(oracle, pts, 3.0, indexed_dims=k, stamp=stamp, reorder=True, ilp=8, shortcircuit=True)
    assert st["join_path"] == 3


@pytest.mark.parametrize("n", [18, 90])
def test_screen_far_and_tight_points(oracle, n):
    """Points 1e16 from the rest (no bound holds there: every pair with them
    takes the exact check) next to cells of exact duplicates, and a second
    cluster whose pairs all lie within eps (32 undecided pairs a record)."""
    pts = tile_points(n, 6000, 3.0, 900 + n)
    pts[7, n - 1] = 1e16
    pts[8, n - 1] = 1e16
    pts[9, n - 2] = -3e18
    pts[1000:1400] = pts[1000]
    pts[2000:2300] = pts[2000] + np.float32(0.01) * np.random.default_rng(1).standard_normal((300, n)).astype(np.float32)
    st = assert_same(oracle, pts, 3.0, indexed_dims=6, stamp=False)
    assert st["join_path"] == 3


@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("n,k,ilp,sc", [(5, 5, 0, False), (6, 2, 8, True), (8, 3, 8, True), (11, 6, 4, False),
                                        (12, 6, 0, False), (13, 6, 8, False), (15, 1, 2, True)])
def test_low_dimensional_screen(oracle, n, k, ilp, sc, stamp):
    """Below 16 dimensions (one MMA step of 16 columns up to n = 12) the tile
    join is screened too and still reports GSJ_PATH_TILE; plain turns it off."""
    pts = tile_points(n, 6003, 3.0, 700 + n)
    st = assert_same(oracle, pts, 3.0, indexed_dims=k, ilp=ilp, shortcircuit=sc, stamp=stamp)
    assert st["join_path"] == 2 and st["screen_rechecks"] > 0
    st = assert_same(oracle, pts, 3.0, indexed_dims=k, ilp=ilp, shortcircuit=sc, stamp=stamp, plain=True)
    assert st["join_path"] == 2 and st["screen_rechecks"] == 0
