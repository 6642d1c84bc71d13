"""The traversals choose per ray between the fast-division form and the general one, and the sampler
culls subtrees behind the origin on cuts that allow it. Every choice against the CPU restatement, bit
for bit: meshes inside the fast domain, outside it (coordinates beyond 2^11), mixed signs with exact
zeros, and rays that leave it one by one (axis-aligned, origins on box planes, tiny components)."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import mesh
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

# scale, offset of the mesh; fixed dilation, extent dilation, learning epsilon, cut depth
FORMS = [
    (1.0, 0.0, 1e-5, 1e-4, 1e-3, 10),
    (2.0, -1.0, 0.0, 0.3, 1e-2, 7),      # zeros and both signs; large random dilations
    (1.0, 4096.0, 1e-5, 1e-4, 1e-3, 6),  # outside the fast-division domain
    (300.0, -7.0, 0.7, 0.6, 0.5, 8),     # dilations above 1: no culling, general division when training
    (1.0, 0.25, 1e-3, 0.0, -1e-3, 30),   # the whole tree; negative epsilons accept segments ending at zero
    (1.0, 0.0, 1e-5, 1e-4, 1e-3, 0),     # the root alone
]


def _scene(form):
    scale, offset, fixed, extent, eps, depth = form
    v, f = mesh("sphere4k", 3)
    v = (v * np.float32(scale) + np.float32(offset)).astype(np.float32)
    cfg = nb.default_config(batch_size=1 << 12, neural_bvh_max_depth=depth)
    b = cfg.bvh
    b.fixed_node_dilation, b.node_extent_dilation = fixed, extent
    b.learning_mint_epsilon = b.learning_maxt_epsilon = eps
    if eps < 0:
        b.inference_mint_epsilon = b.inference_maxt_epsilon = eps
    h = nb.NBVH(cfg)
    h.set_mesh(v, f)
    h.build_classic()
    h.build_neural_cut()
    nodes, prims = h.classic_bvh()
    nn, bbox = h.neural_bvh()
    return h, cfg, v, f, nodes, prims, nn, bbox


def _rays(nn, bbox):
    rays = scenes.uniform_rays(6000, bbox[:3], bbox[3:], seed=9)
    rng = np.random.default_rng(10)
    lo, hi = nb.nodes_to_float(nn)
    k = rng.integers(0, len(nn), 1500)
    rays[:1500, 0:3] = np.where(rng.random((1500, 3)) < 0.5, lo[k], hi[k])  # origins on box planes and corners
    rays[1500:2200, 4:7] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, 700)] * rng.choice([-1, 1], (700, 1))
    rays[2200:2600, 4 + 1] = 0.0
    rays[2600:2800, 4] *= np.float32(1e-30)
    rays[2800:3100, 7] = rng.random(300)  # bounded rays
    rays[3100:3110, 7] = np.nan
    rays[3110:3120, 3] = np.nan
    return np.ascontiguousarray(rays, np.float32)


@pytest.mark.parametrize("form", FORMS)
def test_traversal_forms_match_the_restatement(built, oracle, form):
    h, cfg, v, f, nodes, prims, nn, bbox = _scene(form)
    with h:
        rays = _rays(nn, bbox)
        d_rays = torch.from_numpy(rays).cuda()
        cs = oracle.classic_scene(nodes, prims, v, f)
        got = h.query_closest_classic(d_rays).cpu().numpy().view(np.uint32)
        assert np.array_equal(got, oracle.classic_query(cs, rays).view(np.uint32).reshape(got.shape))
        segs, counts = h.query_segments(d_rays, 16)
        rsegs, rcounts = oracle.neural_segments(nn, oracle.neural_consts(cfg), rays, 16)
        counts = counts.cpu().numpy().view(np.uint32)
        assert np.array_equal(counts, rcounts)
        g, r = segs.cpu().numpy().view(np.uint32), rsegs.view(np.uint32).reshape(-1, 16, 4)
        listed = np.arange(16)[None, :] < np.minimum(counts, 16)[:, None]
        assert np.array_equal(g[listed][:, :3], r[listed][:, :3])
        n = 1 << 12
        pos, tgt, snodes = h.generate_training_batch(5, n)
        rpos, rtgt, rnodes = oracle.training_batch(oracle.neural_scene(nn, bbox), cs, None, oracle.neural_consts(cfg),
                                                   5, cfg.batch_size, n)
        assert np.array_equal(snodes.cpu().numpy().view(np.uint32), rnodes)
        assert np.array_equal(pos.cpu().numpy().view(np.uint32), rpos.view(np.uint32))
        assert np.array_equal(tgt.cpu().numpy().view(np.uint32), rtgt.view(np.uint32))
