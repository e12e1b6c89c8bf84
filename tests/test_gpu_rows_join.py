"""The ROWS path's count and fill kernels: cells of one point up to several
128-candidate groups, the thread-per-query and the cell form of the count pass,
every row width, k = 1..3, double, and the batched host result.  Lists in
candidate order must hold the oracle's neighbours; counts, offsets and the
batched table must agree entry by entry."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin
from tests.test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,k,N,side", [(1, 1, 3001, 900.0), (1, 1, 2000, 7.0), (2, 1, 1500, 40.0),
                                        (2, 2, 4097, 60.0), (2, 2, 4096, 9.0), (3, 2, 3000, 12.0),
                                        (3, 3, 5003, 16.0), (3, 3, 4000, 5.0), (4, 3, 3333, 9.0), (4, 2, 33, 2.0)])
def test_rows_counts_and_lists(oracle, n, k, N, side, dtype):
    rng = np.random.default_rng(n * 100 + k)
    pts = rng.uniform(0, side, size=(N, n))
    pts[: N // 8] = pts[0] + rng.uniform(0, 0.6, size=(N // 8, n))  # one cell of hundreds of points
    pts = pts[rng.permutation(N)].astype(dtype)
    st = assert_same(oracle, pts, 1.0, indexed_dims=k)
    assert st["join_path"] == 1
    with SelfJoin(0) as sj:
        sj.run(pts, 1.0, JoinConfig(indexed_dims=k))
        counts, table = sj.counts(), sj.table()
        _, hc, ht = sj.run_host(pts, 1.0, JoinConfig(indexed_dims=k, buffer_pairs=1, min_batches=5))
    assert np.array_equal(hc, counts) and np.array_equal(ht, table)
