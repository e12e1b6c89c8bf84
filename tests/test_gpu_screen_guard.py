"""The way out of the tensor-core screen.  Below 16 dimensions a bound that decides
nothing (clusters far from the data's mean, a sentinel value that moves it) must
hand the join to the FP32 tiles, undecided pairs that are mostly within eps must
not; at any dimensionality a join whose undecided pairs do not fit the device must
still run.  The lists must be the oracle's exactly."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin
from tests.test_gpu_parity import assert_same, canon

pytestmark = pytest.mark.gpu


def clusters(n, N, spread, seed, K=4):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, spread, size=(K, n))
    return (c[rng.integers(0, K, N)] + 1.5 * rng.standard_normal((N, n))).astype(np.float32)


# some 30 million candidates, all undecided: above the count below which nothing is looked at
@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("n,k,ilp,sc", [(5, 3, 0, False), (8, 3, 8, True), (12, 3, 4, False), (15, 3, 0, False)])
@pytest.mark.parametrize("kind", ["far", "sentinel"])
def test_useless_bound_takes_the_fp32_tiles(oracle, n, k, ilp, sc, stamp, kind):
    eps = 1.2 * n ** 0.5
    pts = clusters(n, 16000, 9000.0 if kind == "far" else 30.0, 40 + n)
    if kind == "sentinel":
        pts[7, n - 1] = 1e9
    st = assert_same(oracle, pts, eps, indexed_dims=k, ilp=ilp, shortcircuit=sc, stamp=stamp)
    assert st["candidates"] > 2 ** 24  # enough of them for the guard to look
    assert st["join_path"] == 2 and st["screen_rechecks"] == 0


@pytest.mark.parametrize("stamp", [False, True])
def test_pairs_within_eps_stay_on_the_screen(oracle, stamp):
    """Four fifths of the candidates are result pairs: undecided, and rightly so."""
    pts = clusters(8, 18000, 30.0, 3)
    st = assert_same(oracle, pts, 2.6 * 8 ** 0.5, indexed_dims=3, stamp=stamp)
    assert st["total_pairs"] > 0.5 * st["candidates"] > 2 ** 23
    assert st["join_path"] == 2 and st["screen_rechecks"] > 2 ** 24


@pytest.mark.parametrize("how", ["learned", "exact_size"])
def test_useless_bound_without_a_sampling_pass(oracle, how):
    eps = 1.2 * 8 ** 0.5
    good, bad = clusters(8, 16000, 30.0, 5), clusters(8, 16000, 9000.0, 6)
    with SelfJoin(0) as sj:
        st = sj.run(good, eps, JoinConfig(indexed_dims=3))
        assert st["screen_rechecks"] > 0
        sj.model_train(200)
        for pts, screened in ((bad, False), (good, True)):
            st = sj.run(pts, eps, JoinConfig(indexed_dims=3, **{how: True}))
            assert (st["screen_rechecks"] > 0) == screened
            oc, _, on = oracle.join_lists(pts, eps, oracle.OracleConfig(k=3))
            assert np.array_equal(sj.counts(), oc) and np.array_equal(canon(sj.counts(), sj.table()), on)
            assert st["candidates"] == oracle.join_counts(pts, eps, oracle.OracleConfig(k=3))[2]


def test_screen_without_room(oracle):
    """2e8 undecided pairs need 1.6 GB as keys; with 1 GB left the FP32 tiles, which
    need room for the result pairs alone, must take the join."""
    import torch

    pts = clusters(18, 40000, 2000.0, 9, K=8)
    eps = 4.0
    oc, _, on = oracle.join_lists(pts, eps, oracle.OracleConfig(k=3))
    with SelfJoin(0) as sj:
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
        try:
            st = sj.run(pts, eps, JoinConfig(indexed_dims=3))
            counts, table = sj.counts(), sj.table()
        finally:
            del hog
            torch.cuda.empty_cache()
        assert st["join_path"] == 2 and st["candidates"] > 1.5e8
        assert np.array_equal(counts, oc) and np.array_equal(canon(counts, table), on)
        st = sj.run(pts, eps, JoinConfig(indexed_dims=3))  # with room again: screened
        assert st["join_path"] == 3 and np.array_equal(sj.counts(), oc)
