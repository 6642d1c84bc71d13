"""The tail kernel deals short lists over all its warps and claims long ones by counter, and takes over
from the wavefront steps earlier the smaller the batch, from the first segment on for the smallest:
its mma.sync tiles and the tcgen05 MLP have to give the same bits. Whole batches against the same rays in pieces, word for word, with
networks that accept about half of the segments and with none accepted (every ray then evaluates
every leaf it enters, as the segment enumeration counts them)."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

# (points, levels, features, precision, hidden layers): a row of a tile is points x levels items of the encoder
NETS = [(4, 16, 2, 0, 4), (3, 8, 4, 1, 4), (2, 4, 8, 2, 4), (1, 8, 2, 0, 1), (4, 16, 2, 1, 8), (4, 8, 4, 2, 3),
        (4, 12, 2, 0, 2), (16, 4, 2, 0, 2), (6, 8, 2, 1, 2)]


@pytest.mark.parametrize("net", NETS)
@pytest.mark.parametrize("threshold", [0.5, 2.0])
def test_tail_lists_of_every_length(built, net, threshold):
    P, L, F, prec, H = net
    cfg = nb.default_config(**{"hashgrid.n_levels": L, "hashgrid.n_features_per_level": F, "hashgrid.base_resolution": 8,
                               "hashgrid.log2_hashmap_size": 14, "module.input_segment_points": P,
                               "network.precision": prec, "network.n_hidden_layers": H,
                               "output.primary_visibility_threshold": threshold})
    h, s = handle(cfg, kind="soup64k", seed=2, depth=12)
    with h:
        rng = np.random.default_rng(5)
        p = h.params()
        nn = h.layout.n_network_params
        p[:nn] *= 2.0
        p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
        h.set_params(p)
        n = 160003  # over 32 rays for every warp of the grid reach the tail when nothing is accepted
        rays = torch.from_numpy(scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=6, scaling=1.0)).cuda()
        whole = h.query_closest_neural(rays)
        segments = whole[:, 9]
        if threshold > 1.0:
            _, counts = h.query_segments(rays, 1)
            assert torch.equal(segments, counts)
            assert int((segments > 5).sum()) > 77824
        for a, size in ((0, 1), (1, 31), (40, 33), (100, 2431), (3000, 2433), (6000, 40001)):
            part = h.query_closest_neural(rays[a:a + size].contiguous())
            assert torch.equal(part, whole[a:a + size]), (a, size)
