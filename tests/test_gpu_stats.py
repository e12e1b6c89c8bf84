"""Host stage times: the index build's share holds all of its device work, and the
stages add up to no more than the call."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,side,eps,kw", [(2, 2, 2000.0, 0.4, {}), (3, 3, 4000.0, 1.0, {}), (6, 6, 12.0, 1.0, {}),
                                             (8, 3, 8.0, 0.5, {}), (2, 2, 2000.0, 0.4, {"sort": True})])
def test_host_stage_times(n, k, side, eps, kw):
    pts = np.random.default_rng(n).uniform(0, side, size=(2_000_000 if n < 6 else 100_000, n)).astype(np.float32)
    with SelfJoin(0) as sj:
        for _ in range(3):
            st = sj.run(pts, eps, JoinConfig(indexed_dims=k, **kw))
            assert st["ms_index"] >= st["dev_ms_index"] > 0
            assert st["ms_join"] >= st["dev_ms_count"] + st["dev_ms_fill"] - 0.05
            assert st["ms_h2d"] + st["ms_index"] + st["ms_join"] <= st["ms_total"] + 0.05
