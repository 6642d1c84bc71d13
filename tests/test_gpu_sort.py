"""The wavefront's counting sort takes a place per row from the bins' cursors or reserves a range per
bin and block, by the list's length against the number of bins. Whole batches (sorted) against the
same rays in pieces below the shortest list that is sorted, word for word: a row placed twice or
not at all would leave a record unwritten or written from another ray's state."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


# cuts of a few, a few hundred and a few thousand nodes; 64 (point, level) pairs: octant bins, 24: none
@pytest.mark.parametrize("points,levels,features", [(4, 16, 2), (3, 8, 4)])
@pytest.mark.parametrize("depth", [2, 7, 10, 12])
def test_sorted_lists_against_unsorted(built, points, levels, features, depth):
    cfg = nb.default_config(**{"hashgrid.n_levels": levels, "hashgrid.n_features_per_level": features,
                               "hashgrid.base_resolution": 8, "hashgrid.log2_hashmap_size": 12,
                               "module.input_segment_points": points})
    h, s = handle(cfg, kind="soup64k", seed=4, depth=depth)
    with h:
        rng = np.random.default_rng(3)
        p = h.params()
        nn = h.layout.n_network_params
        p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
        h.set_params(p)
        # 1,000,003 rays: several rows per thread and a ragged last chunk
        n = 1000003 if depth in (2, 12) else 200001
        rays = torch.from_numpy(scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=5, scaling=1.0)).cuda()
        whole = h.query_closest_neural(rays)
        for a in range(0, n, 65535):
            part = h.query_closest_neural(rays[a:a + 65535].contiguous())
            assert torch.equal(part, whole[a:a + 65535]), a


@pytest.mark.parametrize("depth", [4, 10])
def test_sorted_batch_with_octant_bins(built, depth):
    """600,001 rays: a list of some 4,000 rows per block, fewer than half the bins of the deep cut (places
    straight from the cursors) and more than those of the shallow one (ranges per block)."""
    cfg = nb.default_config(**{"hashgrid.base_resolution": 8, "hashgrid.log2_hashmap_size": 12})
    h, s = handle(cfg, kind="soup64k", seed=4, depth=depth)
    with h:
        rng = np.random.default_rng(3)
        p = h.params()
        nn = h.layout.n_network_params
        p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
        h.set_params(p)
        n = 600001
        rays = torch.from_numpy(scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=6, scaling=1.0)).cuda()
        whole = h.query_closest_neural(rays)
        for a in range(0, n, 65535):
            assert torch.equal(h.query_closest_neural(rays[a:a + 65535].contiguous()), whole[a:a + 65535]), a
