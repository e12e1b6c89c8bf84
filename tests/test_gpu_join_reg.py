"""The warp join's register form: every row width and summation order it is
built for, on sparse cells (a warp's candidates come from many short neighbour
rows) next to one dense blob whose items are cut into slices, hashed and dense
grids.  Lists and, without
unicomp, candidate totals must be the oracle's exactly."""
import numpy as np
import pytest

from tests.test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def mixed(n, k, seed, sparse=9000, dense=5000):
    rng = np.random.default_rng(seed)
    side = 5.0 if k >= 5 else (16.0 if k >= 3 else 400.0)
    x = rng.uniform(0, side, size=(sparse, n))
    x[:, k:] *= 0.3
    blob = rng.uniform(0, 0.9, size=(dense, n)) + 1.3
    blob[:, k:] *= 0.3
    return np.concatenate([x, blob])[rng.permutation(sparse + dense)].astype(np.float32)


# model switches: sequential, one square per register (ILP >= n), blocks of ILP
# with SHORTCIRCUIT, ILP chains (the shared-memory form)
@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("n,k,ilp,sc", [(3, 3, 4, True), (4, 2, 2, True), (4, 4, 0, False), (5, 5, 0, False),
                                        (6, 6, 0, False), (6, 6, 1, True), (7, 6, 8, False), (8, 6, 8, True),
                                        (8, 6, 3, True), (8, 6, 4, False), (9, 6, 16, False), (12, 6, 5, True),
                                        (13, 6, 0, False), (16, 6, 16, True), (16, 5, 7, True), (17, 5, 8, True)])
def test_warp_join_widths(oracle, n, k, ilp, sc, stamp):
    pts = mixed(n, k, 60 + n)
    st = assert_same(oracle, pts, 1.0, indexed_dims=k, ilp=ilp, shortcircuit=sc, stamp=stamp)
    if not stamp:  # the oracle counts the full neighbourhood's evaluations
        ocfg = oracle.OracleConfig(k=k, ilp=ilp, shortcircuit=sc)
        assert st["candidates"] == oracle.join_counts(pts, 1.0, ocfg)[2]
