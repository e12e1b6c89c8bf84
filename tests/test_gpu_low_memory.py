"""Joins on a device with little free memory, from amounts that end them early to
amounts that suffice: each gives the lists it gives with room, or fails for lack of
memory and leaves the context usable.  Lists of thousands of entries, so that a first
try can fail as late as the last buffer, the long lists' second copy."""
import numpy as np
import pytest

from gpu_self_join_b200 import JoinConfig, SelfJoin
from gpu_self_join_b200._native import GsjError
from tests.test_gpu_screen_guard import clusters

pytestmark = pytest.mark.gpu


def sweep(pts, eps, cfg, path, sizes_mb):
    import torch

    with SelfJoin(0) as sj:
        st = sj.run(pts, eps, cfg)
        assert st["join_path"] == path
        counts, table = sj.counts(), sj.table()
    assert counts.max() > 4096
    done = []
    for mb in sizes_mb:
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - mb * 1_000_000, dtype=torch.uint8, device="cuda")
        try:
            with SelfJoin(0) as sj:
                try:
                    sj.run(pts, eps, cfg)
                    assert np.array_equal(sj.counts(), counts) and np.array_equal(sj.table(), table)
                    done.append(mb)
                except GsjError as e:
                    assert "error -3" in str(e)
                    small = sj.run(pts[:2000], eps, cfg)  # the context is usable
                    assert small["total_pairs"] > 0
        finally:
            del hog
            torch.cuda.empty_cache()
    return done


@pytest.mark.parametrize("n,path", [(5, 2), (18, 3)])
def test_screened_joins(n, path):
    pts = clusters(n, 24000, 30.0, 2, K=4)
    sizes = [100, 200, 300, 400, 500, 600, 700, 800, 1000, 1200, 1500, 1800, 2200, 2700, 3500, 6000]
    done = sweep(pts, 2.2 * n ** 0.5, JoinConfig(indexed_dims=3, stamp=True), path, sizes)
    assert sizes[-1] in done
