"""The warp join on hashed grids of one to three indexed dimensions, whose
neighbour rows are looked up by a kernel of their own from 32,768 cells on: rows of
one cell and of hundreds, cells at every edge of the grid, more dimensions than
indexed ones.  Lists and, without unicomp, candidate totals
must be the oracle's exactly."""
import numpy as np
import pytest

from tests.test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def hashed(n, k, N, seed, crowd=None):
    """Extents of 25 million cells of side 1 (beyond the dense limit of 2^24): long rows
    along dim 0, a crowded corner, the eight corners of the grid."""
    rng = np.random.default_rng(seed)
    ext = {1: [2.5e7], 2: [5000.0, 5000.0], 3: [6250.0, 80.0, 50.0]}[k]
    x = rng.uniform(0, 1, size=(N, k)) * ext
    x[: N // 4, 0] = rng.uniform(0, 300.0, N // 4)       # rows of hundreds of cells
    x[: N // 4, 1:] = rng.integers(0, 4, size=(N // 4, k - 1)) + 0.5
    crowd = N // 2 - N // 4 if crowd is None else crowd
    x[N // 4: N // 4 + crowd] = rng.uniform(0, 6.0, size=(crowd, k))
    x[-8:] = np.array([[(c >> j) & 1 for j in range(k)] for c in range(8)]) * ext
    return np.concatenate([x, 0.4 * rng.uniform(0, 1, size=(N, n - k))], 1)[rng.permutation(N)]


@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("dtype,n,k,N,ilp", [(np.float64, 1, 1, 3001, 0), (np.float64, 2, 2, 4096, 0), (np.float64, 3, 3, 4099, 0),
                                             (np.float64, 5, 2, 2000, 3), (np.float32, 2, 2, 129, 0), (np.float32, 2, 2, 5001, 2),
                                             (np.float32, 3, 3, 4000, 0), (np.float32, 6, 3, 3003, 0),
                                             (np.float32, 17, 3, 1500, 4)])
def test_hashed_low_dimensional_grids(oracle, dtype, n, k, N, ilp, stamp):
    pts = hashed(n, k, N, 10 * n + k).astype(dtype)
    st = assert_same(oracle, pts, 1.0, indexed_dims=k, ilp=ilp, stamp=stamp)
    assert st["join_path"] == 0 and st["total_cells"] > 1 << 24
    if not stamp:
        assert st["candidates"] == oracle.join_counts(pts, 1.0, oracle.OracleConfig(k=k, ilp=ilp))[2]


# around 32,768 cells: just below (looked up in the join), and the plan's last block of
# 128 cells full, one over and partly filled
@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("dtype,n,k,cells,ilp", [(np.float64, 1, 1, 32767, 0), (np.float64, 1, 1, 32768, 0), (np.float64, 2, 2, 32769, 0),
                                                 (np.float64, 3, 3, 33000, 0), (np.float64, 5, 2, 32896, 3), (np.float32, 2, 2, 32768, 0),
                                                 (np.float32, 3, 3, 32767, 0), (np.float32, 3, 3, 32897, 0),
                                                 (np.float32, 6, 3, 40000, 0), (np.float32, 17, 3, 33333, 4)])
def test_plan_line(oracle, dtype, n, k, cells, ilp, stamp):
    pts = hashed(n, k, 4 * cells // 2, 5 * n + k, crowd=500).astype(dtype)
    # whole cells are taken away until that many are left (not those at the extremes)
    key = np.floor((pts[:, :k] - (pts[:, :k].min(0) - dtype(1.0))) / dtype(1.0)).astype(np.int64)
    uniq, cell = np.unique(key, axis=0, return_inverse=True)
    cell = cell.reshape(-1)
    ends = np.unique(cell[np.concatenate([pts[:, :k].argmin(0), pts[:, :k].argmax(0)])])
    rest = np.setdiff1d(np.random.default_rng(1).permutation(len(uniq)), ends, assume_unique=True)
    keep = np.concatenate([ends, rest])[:cells]
    assert keep.size == cells
    pts = np.ascontiguousarray(pts[np.isin(cell, keep)])
    st = assert_same(oracle, pts, 1.0, indexed_dims=k, ilp=ilp, stamp=stamp)
    assert st["join_path"] == 0 and st["total_cells"] > 1 << 24 and st["nonempty_cells"] == cells
    if not stamp:
        assert st["candidates"] == oracle.join_counts(pts, 1.0, oracle.OracleConfig(k=k, ilp=ilp))[2]
