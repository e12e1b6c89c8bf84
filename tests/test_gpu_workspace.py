"""Device memory that a small join of the pair-emitting paths takes: the room for the
warps' partly filled blocks is sized by the warps that are launched."""
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


# Warp join: at most 32 resident warps an SM in each of its two launches, a block of 1,024
# keys of 8 bytes each, buffers half as large again: 148 x 64 x 1024 x 8 x 1.5 = 117 MB,
# 13 MB for the list of slices, the rest below 20.  Screen: 148 x 16 warps, 256 records of
# 16 bytes: 15 MB, the rest below 25.
@pytest.mark.parametrize("n,k,path,limit", [(6, 6, 0, 150e6), (8, 3, 2, 40e6), (18, 3, 3, 40e6)])
def test_workspace_of_small_joins(n, k, path, limit):
    rng = np.random.default_rng(n)
    pts = rng.uniform(0, 20.0 if path == 0 else 6.0, size=(8000, n)).astype(np.float32)
    got, st = taken(pts, 1.0, indexed_dims=k)
    assert st["join_path"] == path
    assert got < limit
