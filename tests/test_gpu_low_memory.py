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
        with SelfJoin(0) as sj:
            try:
                sj.run(pts, eps, cfg)
                assert np.array_equal(sj.counts(), counts) and np.array_equal(sj.table(), table)
                done.append(mb)
            except GsjError as e:
                assert "error -3" in str(e)
            finally:
                del hog
                torch.cuda.empty_cache()
            # with room again the same context joins
            st = sj.run(pts[:2000], eps, cfg)
            assert st["total_pairs"] == int(sj.counts().sum(dtype=np.uint64)) > 0
    return done


@pytest.mark.parametrize("n,path", [(5, 2), (18, 3)])
def test_screened_joins(n, path):
    pts = clusters(n, 24000, 30.0, 2, K=4)
    sizes = [100, 200, 300, 400, 500, 600, 700, 800, 1000, 1200, 1500, 1800, 2200, 2700, 3500, 6000]
    done = sweep(pts, 2.2 * n ** 0.5, JoinConfig(indexed_dims=3, stamp=True), path, sizes)
    assert sizes[-1] in done


def test_joins_with_a_row_plan():
    """A hashed 3-D grid in double: 72 bytes of row plan a cell, which the join gives up
    before it fails."""
    rng = np.random.default_rng(3)
    pts = rng.uniform(0, 2000.0, size=(800_000, 3))
    pts[:9000] = 1000.0 + rng.uniform(0, 0.9, size=(9000, 3))
    sizes = [60, 100, 150, 200, 230, 260, 290, 320, 350, 380, 420, 460, 500, 560, 640, 740, 900, 1200, 2500]
    done = sweep(pts, 1.0, JoinConfig(indexed_dims=3), 0, sizes)
    assert sizes[-1] in done
