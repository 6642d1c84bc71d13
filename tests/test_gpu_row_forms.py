"""Encoding and gradient scatter of explicit rows: one thread per point or its levels spread over
several, stores of 16 bytes or less, points of a row merged while they stay in one cell. Sizes where
the choices change and where blocks end, against the stand-alone encoder and the CPU restatement."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import check_gradients

pytestmark = pytest.mark.gpu

# (points, levels, features): every store width, level counts that are no multiple of a store
GRIDS = [(4, 16, 2), (4, 6, 2), (2, 12, 4), (4, 1, 4), (2, 3, 8), (1, 16, 8)]


def _handle(grid, precision=0):
    P, L, F = grid
    cfg = nb.default_config(**{"hashgrid.n_levels": L, "hashgrid.n_features_per_level": F, "hashgrid.base_resolution": 4,
                               "hashgrid.per_level_scale": 1.7, "hashgrid.log2_hashmap_size": 12,
                               "module.input_segment_points": P, "network.precision": precision})
    h = nb.NBVH(cfg)
    rng = np.random.default_rng(3)
    p = h.params()
    nn = h.layout.n_network_params
    p[:nn] *= 2.0
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    h.set_params(p)
    return h, p


def _rows(n, P, seed):
    """Rows of points close together (most share a coarse cell), the cube's border among them."""
    rng = np.random.default_rng(seed)
    a = rng.random((n, 1, 3))
    pos = a + rng.uniform(-0.05, 0.05, (n, 1, 3)) * (np.arange(P)[None, :, None] - rng.integers(0, 2, (n, 1, 1)))
    pos[: n // 8] = np.round(pos[: n // 8])
    return np.clip(pos, 0.0, 1.0).astype(np.float32)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("n", [1, 31, 129, 40000])
def test_rows_match_the_encoder_and_mlp(built, grid, n):
    h, _ = _handle(grid)
    with h:
        pos = torch.from_numpy(_rows(n, grid[0], n)).cuda()
        want = h.mlp_inference(h.encode(pos).half())  # the same rounding of the same FP32 features
        assert torch.equal(h.network_inference(pos), want)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("n", [1, 33, 700])
def test_gradients_of_merged_points(built, oracle, grid, n):
    h, p = _handle(grid)
    with h:
        pos = _rows(n, grid[0], 5 + n)
        rng = np.random.default_rng(n)
        tgt = rng.random((n, 8)).astype(np.float32)
        tgt[:, 0] = tgt[:, 0] < 0.6
        g, loss = h.compute_gradients(torch.from_numpy(pos).cuda(), torch.from_numpy(tgt).cuda())
        rg, rloss = oracle.compute_gradients(oracle.network(h.cfg, h.layout, p), oracle.loss_consts(h.cfg), pos, tgt,
                                             h.layout.n_params, loss_scale=h.cfg.optimizer.loss_scale)
        assert abs(loss - rloss) <= 1e-3 * abs(rloss) + 1e-6
        check_gradients(oracle, h, p, pos, tgt, g.cpu().numpy().astype(np.float64), rg.astype(np.float64), 2e-2)


@pytest.mark.parametrize("scale", [128.0, 100.0])
def test_gradient_buffers_and_loss_scales(built, oracle, scale):
    """A buffer the kernels can add into, one off 16 bytes and one that holds the targets get the same
    gradient up to the order of its float additions; a loss scale that is no power of two as well."""
    h0, p = _handle((4, 16, 2))
    h0.close()
    h0.cfg.optimizer.loss_scale = scale
    with nb.NBVH(h0.cfg) as h:
        h.set_params(p)
        n = 700
        pos, rng = _rows(n, 4, 8), np.random.default_rng(8)
        tgt = rng.random((n, 8)).astype(np.float32)
        d_pos, d_tgt = torch.from_numpy(pos).cuda(), torch.from_numpy(tgt).cuda()
        g, loss = h.compute_gradients(d_pos, d_tgt)
        rg, _ = oracle.compute_gradients(oracle.network(h.cfg, h.layout, p), oracle.loss_consts(h.cfg), pos, tgt,
                                         h.layout.n_params, loss_scale=scale)
        check_gradients(oracle, h, p, pos, tgt, g.cpu().numpy().astype(np.float64), rg.astype(np.float64), 2e-2)
        big = torch.zeros(h.layout.n_params + 1, device="cuda")
        for off, targets in ((1, d_tgt), (0, big[:n * 8])):
            if targets is not d_tgt:
                targets.copy_(d_tgt.view(-1))
            assert h.lib.nbvh_compute_gradients(h.h, nb._ptr(d_pos), nb._ptr(targets), n, nb._ptr(big[off:]), None,
                                                nb._stream(None)) == 0
            # addends of one sign scale, thousands of them at most: far below 1e-4 of the largest
            assert (big[off:off + g.numel()] - g).abs().max() <= 1e-4 * g.abs().max()
