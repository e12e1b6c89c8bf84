"""The sampled variance statistic behind reordered dimensions: dimension counts
around a block's 8, sample counts around the staged chunk (992 samples of
FP32, 496 of FP64).  The order of the dimensions hangs on single sampled rows
(an outlier column by column at the first and last row of every chunk) and, for
columns holding the same values in another order, on the rounding of the
sequential sums; lists, cells and candidates must be those of the oracle's order."""
import numpy as np
import pytest

from tests.test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nsamp,dtype", [(1, 1, np.float32), (2, 16, np.float32), (7, 17, np.float64),
                                           (8, 496, np.float64), (9, 497, np.float64), (8, 992, np.float32),
                                           (9, 993, np.float32), (17, 1985, np.float32)])
def test_variance_order(oracle, n, nsamp, dtype):
    rng = np.random.default_rng(nsamp * 31 + n)
    N = 100 * nsamp - 37 if nsamp > 1 else 60
    chunk = 992 if dtype == np.float32 else 496
    x = rng.uniform(0, 40, size=(N, n)).astype(dtype)  # only the sampled rows enter the statistic
    rows = np.arange(0, N, 100)
    base = rng.uniform(0, 1, size=rows.size).astype(dtype)
    for j in range(n):  # the same sampled values in every column, shuffled
        x[rows, j] = base[rng.permutation(rows.size)]
    edge = sorted({0, chunk - 1, chunk, 2 * chunk - 1, 2 * chunk, rows.size - 1} & set(range(rows.size)))
    for i, s in enumerate(edge[: max(n - 2, 0)]):  # one outlier each, in columns from the last
        x[100 * s, n - 1 - i] = dtype(3.0 + 0.5 * i)
    k = min(n, 3)
    eps = 1.0 if n > 2 else 0.25
    st = assert_same(oracle, x, eps, indexed_dims=k, reorder=True)
    perm, _ = oracle.reorder_perm(x)
    _, _, _, total = oracle.grid_dims(x[:, perm], k, eps)
    assert st["total_cells"] == total
    assert st["candidates"] == oracle.join_counts(x, eps, oracle.OracleConfig(k=k, reorder=True))[2]
