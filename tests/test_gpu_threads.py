"""Two contexts in two threads whose joins use the same kernels with different
amounts of shared memory: every join must launch and give the lists it gives
alone."""
import threading

import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin
from tests.test_gpu_parity import tile_points

pytestmark = pytest.mark.gpu


# screen (18 and 120 dims), FP32 tiles (8 and 128), warp join (2 of 3 and 7 of 7 dims indexed, double)
@pytest.mark.parametrize("path,a,b", [
    (3, dict(n=18, k=3), dict(n=120, k=6)),
    (2, dict(n=8, k=3, plain=True), dict(n=128, k=6, plain=True)),
    (0, dict(n=6, k=2, ilp=3, dtype=np.float64), dict(n=7, k=7, ilp=2, dtype=np.float64)),
])
def test_two_contexts_two_sizes(path, a, b):
    errors = []
    start = threading.Barrier(2)

    def work(n, k, dtype=np.float32, **kw):
        try:
            pts = tile_points(n, 3000, 3.0, 70 + n).astype(dtype)
            cfg = JoinConfig(indexed_dims=k, **kw)
            with SelfJoin(0) as sj:
                st = sj.run(pts, 3.0, cfg)
                assert st["join_path"] == path
                counts = sj.counts()
                start.wait(60)
                for i in range(200):
                    sj.run(pts, 3.0, cfg)
                    if i % 50 == 0:
                        assert np.array_equal(sj.counts(), counts)
        except Exception as e:  # reported by the main thread
            start.abort()
            errors.append(repr(e))

    threads = [threading.Thread(target=work, kwargs=kw) for kw in (a, b)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
