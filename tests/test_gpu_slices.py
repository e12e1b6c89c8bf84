"""The warp join's slice list: long items cut into slices, a list that is full
after some of them (or from the start), counters beyond 32 bits.  The lists must
be the oracle's whatever the list holds."""
import ctypes

import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin, _native
from tests.test_gpu_join_reg import mixed
from tests.test_gpu_parity import canon

pytestmark = pytest.mark.gpu


def hook(sj, cap, before):
    found = ctypes.c_uint64()
    _native.check(_native.lib().gsj_test_slice_list(sj._ctx, cap, before, ctypes.byref(found)), sj._ctx)
    return found.value


# capacities: the built-in one, one that an item overflows part way, one slice; counts
# from 0, from a full list, and across 2^32 (a 32-bit counter would start over)
@pytest.mark.parametrize("stamp", [False, True])
@pytest.mark.parametrize("n,ilp", [(6, 0), (8, 8), (13, 0)])
def test_slice_list_capacity_and_count(oracle, n, ilp, stamp):
    pts = mixed(n, 6, 300 + n, sparse=4000, dense=6000)
    oc, _, on = oracle.join_lists(pts, 1.0, oracle.OracleConfig(k=6, ilp=ilp, shortcircuit=ilp > 0))
    cfg = JoinConfig(indexed_dims=6, ilp=ilp, shortcircuit=ilp > 0, stamp=stamp)
    with SelfJoin(0) as sj:
        slices = None
        for cap, before in ((0, 0), (101, 0), (1, 0), (0, 1 << 20), (257, (1 << 32) - 3)):
            hook(sj, cap, before)
            st = sj.run(pts, 1.0, cfg)
            assert st["join_path"] == 0  # GSJ_PATH_WARP
            assert np.array_equal(sj.counts(), oc) and np.array_equal(canon(sj.counts(), sj.table()), on)
            found = hook(sj, 0, 0) - before
            if slices is None:
                slices = found
            assert found == slices > 257
    assert int(oc.sum()) == on.size
