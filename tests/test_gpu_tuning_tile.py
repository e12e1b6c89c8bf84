"""GSJ_PATH_TILE stands for the screen and for the FP32 tiles below 16 dimensions: a
shape tuned on one must not shape the other, an entry set by hand applies to both."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin
from tests.test_gpu_parity import tile_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuned_plain", [False, True])
def test_screened_and_plain_tile_shapes_are_apart(tuned_plain):
    pts = tile_points(12, 8000, 3.0, 12)
    cfgs = {p: JoinConfig(indexed_dims=6, plain=p) for p in (False, True)}
    with SelfJoin(0) as sj:
        st = sj.run(pts, 3.0, cfgs[False])
        counts, table = sj.counts(), sj.table()
        assert st["join_path"] == 2 and st["screen_rechecks"] > 0 and st["tuned"] == 0
        key = (2, 12, int(st["density_log2"]))
        best = sj.autotune(pts, 3.0, cfgs[tuned_plain], repeats=1)
        assert sj.tuning(*key) == best
        for plain in (False, True):
            st = sj.run(pts, 3.0, cfgs[plain])
            assert st["tuned"] == (plain == tuned_plain)
            assert np.array_equal(sj.counts(), counts) and np.array_equal(sj.table(), table)
        assert sj.tuning(*key, {"ctas_per_sm": 1})["ctas_per_sm"] == 1
        for plain in (False, True):
            st = sj.run(pts, 3.0, cfgs[plain])
            assert st["tuned"] == 1
            assert np.array_equal(sj.counts(), counts) and np.array_equal(sj.table(), table)
