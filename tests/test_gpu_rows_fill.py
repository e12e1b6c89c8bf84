"""The ROWS path's three fill forms on both sides of the lines between them: a
thread per query (sparse cells, short lists), the cell form, and the cell form for
candidates of which few are within eps.  The lists must be the oracle's, in the
order of the batched host result."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin
from tests.test_gpu_parity import canon

pytestmark = pytest.mark.gpu


def check(oracle, pts, k):
    oc, _, on = oracle.join_lists(pts, 1.0, oracle.OracleConfig(k=k))
    with SelfJoin(0) as sj:
        st = sj.run(pts, 1.0, JoinConfig(indexed_dims=k))
        counts, table = sj.counts(), sj.table()
        _, hc, ht = sj.run_host(pts, 1.0, JoinConfig(indexed_dims=k, buffer_pairs=1, min_batches=4))
    assert st["join_path"] == 1
    assert np.array_equal(counts, oc) and np.array_equal(canon(counts, table), on)
    assert np.array_equal(hc, counts) and np.array_equal(ht, table)
    return st


# points a cell (of the whole grid) from far below to above the lines at 5 and 7 points
# a non-empty cell; pairs a point from 1 to beyond 5 + 3^(k-1)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,k,density", [(1, 1, 0.4), (1, 1, 2.5), (1, 1, 4.0), (2, 2, 0.05), (2, 2, 1.0), (2, 2, 2.2),
                                         (2, 2, 4.5), (2, 2, 6.5), (3, 3, 0.3), (3, 3, 2.0), (3, 3, 4.0),
                                         (4, 3, 1.5), (4, 3, 4.0), (3, 2, 1.0), (2, 1, 3.0), (4, 2, 3.0)])
def test_sparse_cells(oracle, n, k, density, dtype):
    rng = np.random.default_rng(int(100 * density) + 10 * n + k)
    N = 6007
    pts = rng.uniform(0, (N / density) ** (1.0 / k), size=(N, n))
    pts[:, k:] *= 0.01
    pts[100:140] = pts[99]  # one cell with a list longer than a warp
    check(oracle, pts.astype(dtype), k)


# one candidate in some 40 to several hundred within eps: both sides of 1 in 64 (float)
# and 1 in 256 (double)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,k,N,side,other", [(2, 1, 4001, 40.0, 50.0), (3, 1, 3003, 20.0, 10.0), (3, 2, 5001, 9.0, 900.0),
                                              (4, 2, 5003, 5.0, 5.0), (4, 3, 6001, 3.0, 60.0), (4, 1, 2049, 2.0, 40.0)])
def test_few_candidates_within_eps(oracle, n, k, N, side, other, dtype):
    rng = np.random.default_rng(N + n)
    pts = np.concatenate([rng.uniform(0, side, size=(N, k)), rng.uniform(0, other, size=(N, n - k))], 1)
    pts[50:90] = pts[49] + rng.uniform(0, 0.2, size=(40, n))  # some queries with long lists among them
    st = check(oracle, pts.astype(dtype), k)
    assert st["total_pairs"] * 30 < st["candidates"]
