"""Every form of the wavefront's counting sort on lists long enough to be sorted: with and without octant
bins, places taken straight from the bins' cursors (a chunk has at most half as many rows as there
are bins) and ranges reserved per bin, up to the list of a 2^22-ray query. Whole batches against the
same rays in pieces that are too small to be sorted, word for word; the launch count shows that the
sorts ran."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

MIN_RAYS, MIN_ROWS = 1 << 19, 1 << 17  # of a batch whose lists are sorted, of a list that is


def _model(points, levels, features, kind, depth):
    cfg = nb.default_config(**{"hashgrid.n_levels": levels, "hashgrid.n_features_per_level": features,
                               "hashgrid.base_resolution": 8, "hashgrid.log2_hashmap_size": 12,
                               "module.input_segment_points": points})
    h, s = handle(cfg, kind=kind, seed=4, depth=depth)
    rng = np.random.default_rng(3)
    p = h.params()
    nn = h.layout.n_network_params
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    h.set_params(p)
    return h, s


def _check(h, rays, steps):
    n = rays.shape[0]
    whole = h.query_closest_neural(rays)
    # begin, first pass, two for the ray order; per step sort, encoder, MLP, decode; sort and tail
    assert h.last_kernel_time()[1] == 4 + 4 * steps + 2
    assert int((whole[:, 9] > 0).sum()) >= MIN_ROWS
    for a in range(0, n, MIN_RAYS - 1):
        part = rays[a:a + MIN_RAYS - 1].contiguous()
        assert torch.equal(h.query_closest_neural(part), whole[a:a + MIN_RAYS - 1]), a


# (points, levels, features): 64 (point, level) pairs have octant bins, 24 have none. Rows: all rays enter the
# box, or 140,000 do, some 920 rows per block. Nodes: 7, 255, 2,047, 4,095, 8,191 (and 8 times as many bins)
@pytest.mark.parametrize("net", [(4, 16, 2), (3, 8, 4)])
@pytest.mark.parametrize("depth", [2, 7, 10, 11, 12])
@pytest.mark.parametrize("rows", [0, 140000])
def test_sorted_against_unsorted(built, net, depth, rows):
    h, s = _model(*net, "soup64k", depth)
    with h:
        n = 530001
        rays = scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=5, scaling=1.0)
        if rows:  # the others start far away and point away
            away = np.random.default_rng(8).permutation(n)[rows + rows // 50:]
            rays[away, 0:3], rays[away, 4:7] = 1.0e3, 0.57735026
        _check(h, torch.from_numpy(rays).cuda(), 4)


def test_largest_list(built):
    """2^22 rays on the 1,024-leaf cut with octant bins: 16,376 bins, over 1.2 million rows in the first list."""
    h, s = _model(4, 16, 2, "sphere65k", 10)
    with h:
        assert 8 * len(s["neural"]) > 16000
        rays = torch.from_numpy(scenes.uniform_rays(1 << 22, s["bbox"][:3], s["bbox"][3:], seed=6)).cuda()
        _check(h, rays, 5)
        assert int((h.query_closest_neural(rays)[:, 9] > 0).sum()) > 1200000
