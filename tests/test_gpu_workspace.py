"""Buffers of small joins on the pair-emitting paths: no more room for the warps' partly
filled blocks than they can need, and enough of it that a coarse estimate repeats no
pass."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin

pytestmark = pytest.mark.gpu


def taken(pts, eps, **kw):
    import torch

    with SelfJoin(0) as sj:  # loads the kernels
        st = sj.run(pts, eps, JoinConfig(**kw))
    with SelfJoin(0) as sj:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        sj.run(pts, eps, JoinConfig(**kw))
        return free - torch.cuda.mem_get_info()[0], st


# At most 32 resident warps an SM in each of the warp join's two launches, a block of 1,024
# keys of 8 bytes each, buffers half as large again: 148 x 64 x 1024 x 8 x 1.5 = 117 MB,
# 13 MB for the list of slices, the rest below 20.
def test_workspace_of_a_small_warp_join():
    pts = np.random.default_rng(6).uniform(0, 20.0, size=(8000, 6)).astype(np.float32)
    got, st = taken(pts, 1.0, indexed_dims=6)
    assert st["join_path"] == 0
    assert got < 150e6


def test_small_joins_are_not_repeated():
    """6,000 points in four far clusters: a sample of 7 items says 2.6 million undecided
    pairs, there are 8.8 million."""
    from tests.test_gpu_screen_guard import clusters

    for n, k in ((15, 6), (12, 6), (8, 3), (18, 6)):
        pts = clusters(n, 6000, 9000.0, 1)
        with SelfJoin(0) as sj:
            assert sj.run(pts, 1.2 * n ** 0.5, JoinConfig(indexed_dims=k))["reruns"] == 0
