"""The SORT path on hashed grids: neighbour cells found through their grid row, rows
of one cell and of hundreds, cells at the grid's edges.  Lists and candidate
totals must be the oracle's exactly."""
import numpy as np
import pytest

from tests.test_gpu_row_plan import hashed
from tests.test_gpu_sort import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,k,ilp,sc", [(np.float64, 1, 1, 0, False), (np.float64, 2, 2, 0, False), (np.float32, 2, 2, 0, False),
                                              (np.float32, 3, 3, 2, True), (np.float64, 4, 3, 0, False),
                                              (np.float32, 5, 2, 4, False), (np.float32, 18, 3, 8, True)])
def test_sort_on_hashed_grids(oracle, dtype, n, k, ilp, sc):
    pts = hashed(n, k, 4001, 90 + 10 * n + k).astype(dtype)
    st = check(oracle, pts, 1.0, k, ilp=ilp, sc=sc)
    assert st["total_cells"] > 1 << 24


def test_sort_on_a_hashed_six_dimensional_grid(oracle):
    rng = np.random.default_rng(5)
    pts = np.concatenate([rng.uniform(0, 40, size=(3000, 7)), 20 + rng.uniform(0, 2, size=(2000, 7))])
    st = check(oracle, pts.astype(np.float32), 1.0, 6, ilp=8, sc=True)
    assert st["total_cells"] > 1 << 24
