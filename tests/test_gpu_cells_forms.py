"""The wavefront encoder's features from the cell copy of the coarse levels against those from the table
alone: the same records, word for word, for every number of features per level, precision and segment
distribution, and for copies that end anywhere in the grid."""

import ctypes as C

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

N = 1 << 20  # the second query of this size on one set of parameters builds the copy


def _allocations():
    n = C.c_uint64(0)
    assert nb.load_library().nbvh_debug_alloc_count(C.byref(n)) == abi.NBVH_OK
    return n.value


# points, levels, features, precision, segment distribution; hashed and dense levels in each
FORMS = [(4, 16, 2, 0, 0), (4, 16, 2, 1, 2), (2, 8, 2, 2, 1), (4, 4, 2, 0, 0), (3, 8, 4, 0, 0), (4, 5, 4, 1, 1),
         (4, 7, 4, 2, 2), (4, 4, 8, 0, 0), (2, 7, 8, 1, 2), (16, 1, 8, 2, 0), (5, 2, 8, 0, 1)]


@pytest.mark.parametrize("form", FORMS)
def test_copy_against_table(built, form):
    P, L, F, precision, distribution = form
    cfg = nb.default_config(**{"hashgrid.n_levels": L, "hashgrid.n_features_per_level": F, "hashgrid.base_resolution": 8,
                               "hashgrid.per_level_scale": 1.5, "hashgrid.log2_hashmap_size": 14,
                               "module.input_segment_points": P, "module.segment_distribution": distribution,
                               "network.precision": precision})
    h, s = handle(cfg, kind="soup64k", seed=2, depth=10)
    with h:
        rng = np.random.default_rng(5)
        p = h.params()
        nn = h.layout.n_network_params
        p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
        h.set_params(p)
        rays = torch.from_numpy(scenes.uniform_rays(N, s["bbox"][:3], s["bbox"][3:], seed=6, scaling=1.0)).cuda()
        h.set_cell_copy(0)
        table = h.query_closest_neural(rays)
        hits = int((table[:, 8] & 1).sum())
        assert N // 20 < hits < N
        # 8 (F = 2) or 7 levels at most, 4 to 6, 3 or 4, none
        for size in (192 << 20, 32 << 20, 1 << 20, 1 << 10):
            h.set_cell_copy(size)
            h.query_closest_neural(rays)
            before = _allocations()
            for _ in range(2):
                assert torch.equal(h.query_closest_neural(rays), table), size
            assert _allocations() == before + (1 if size > 1 << 10 else 0), size
        # uniform points are drawn by the ray's index in its batch: the first piece alone has the same
        n = 1 << 14 if distribution == 2 else 1 << 16
        small = torch.cat([h.query_closest_neural(r) for r in rays[:n].split(1 << 14)])
        assert torch.equal(small, table[:n])
