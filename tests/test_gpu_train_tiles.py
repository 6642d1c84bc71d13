"""The training kernel over several tiles per block: the tile ahead copied in pieces of 8 rows x 64 bytes
(input widths that are no multiple of that), layer 0 with an accumulator of its own or shared (the hidden
layer count decides), batches in one pass or several. A batch against its two halves, each of one tile per
block: BF16 keeps the factor 2 between their loss normalisations exact, so only the order of the FP32
sums differs, far below 1e-4 of the largest gradient for thousands of addends of one scale."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import check_gradients

pytestmark = pytest.mark.gpu


def _handle(points, hidden, precision, levels=8, features=2):
    cfg = nb.default_config(**{"hashgrid.n_levels": levels, "hashgrid.n_features_per_level": features,
                               "hashgrid.base_resolution": 4,
                               "hashgrid.per_level_scale": 1.5, "hashgrid.log2_hashmap_size": 12,
                               "module.input_segment_points": points, "network.precision": precision,
                               "network.n_hidden_layers": hidden})
    h = nb.NBVH(cfg)
    rng = np.random.default_rng(6)
    p = h.params()
    nn = h.layout.n_network_params
    p[:nn] *= 2.0
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    h.set_params(p)
    return h, p


def _batch(n, points, seed):
    rng = np.random.default_rng(seed)
    tgt = rng.random((n, 8)).astype(np.float32)
    tgt[:, 0] = tgt[:, 0] < 0.6
    return rng.random((n, points, 3)).astype(np.float32), tgt


@pytest.mark.parametrize("points", [1, 3, 5, 7, 8])  # 16, 48, 80, 112, 128 inputs
@pytest.mark.parametrize("hidden", [1, 4, 5, 8])
def test_batch_equals_its_halves(built, points, hidden):
    h, _ = _handle(points, hidden, 1)
    with h:
        m = 19391  # 151 tiles and a ragged one; twice that: two tiles for every block
        pos, tgt = (torch.from_numpy(x).cuda() for x in _batch(2 * m, points, points * 10 + hidden))
        g, loss = h.compute_gradients(pos, tgt)
        parts = [h.compute_gradients(pos[a:a + m].contiguous(), tgt[a:a + m].contiguous()) for a in (0, m)]
        want = (parts[0][0].double() + parts[1][0].double()) / 2
        assert torch.isfinite(g).all() and (want != 0).any()
        assert (g.double() - want).abs().max() <= 1e-4 * want.abs().max()
        assert abs(loss - (parts[0][1] + parts[1][1]) / 2) <= 1e-4 * abs(loss)


@pytest.mark.parametrize("points,levels,features", [(4, 16, 2), (3, 8, 4), (1, 2, 8)])
def test_ordered_batch_equals_its_halves(built, points, levels, features):
    """From 196,608 rows on a batch is encoded in the order of its rows' places, its halves in batch order."""
    h, _ = _handle(points, 2, 1, levels, features)
    with h:
        m = 98305
        pos, tgt = _batch(2 * m, points, points)
        pos[: m // 4] = np.round(pos[: m // 4])  # the cube's border
        pos[m:m + 50] = 0.25  # more rows in one place than a warp has lanes
        pos, tgt = torch.from_numpy(pos).cuda(), torch.from_numpy(tgt).cuda()
        g, loss = h.compute_gradients(pos, tgt)
        parts = [h.compute_gradients(pos[a:a + m].contiguous(), tgt[a:a + m].contiguous()) for a in (0, m)]
        want = (parts[0][0].double() + parts[1][0].double()) / 2
        assert torch.isfinite(g).all() and (want != 0).any()
        assert (g.double() - want).abs().max() <= 1e-4 * want.abs().max()
        assert abs(loss - (parts[0][1] + parts[1][1]) / 2) <= 1e-4 * abs(loss)


@pytest.mark.parametrize("points,hidden", [(3, 1), (7, 5)])
def test_odd_widths_against_the_restatement(built, oracle, points, hidden):
    h, p = _handle(points, hidden, 0)
    with h:
        pos, tgt = _batch(300, points, 9)
        g, loss = h.compute_gradients(torch.from_numpy(pos).cuda(), torch.from_numpy(tgt).cuda())
        rg, rloss = oracle.compute_gradients(oracle.network(h.cfg, h.layout, p), oracle.loss_consts(h.cfg), pos, tgt,
                                             h.layout.n_params, loss_scale=h.cfg.optimizer.loss_scale)
        assert abs(loss - rloss) <= 1e-3 * abs(rloss) + 1e-6
        check_gradients(oracle, h, p, pos, tgt, g.cpu().numpy().astype(np.float64), rg.astype(np.float64), 2e-2)
