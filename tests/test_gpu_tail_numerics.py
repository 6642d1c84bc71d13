"""A segment's outputs come from the wavefront's tcgen05 MLP or from the tail kernel's mma.sync tiles, by
the size of the batch the ray came in. Both have to give the same bits on every network a program may
hold, also where the order and the width of an accumulator would show: sums over a wide range of
exponents, sums that cancel, activations at the FP16 limit and beyond it, subnormal ones, saturated
outputs. Whole batches (their first segments through tcgen05) against the same rays in pieces that the
tail kernel answers alone, word for word; with a threshold below zero every ray's record holds the
outputs of its first segment (of the first that is no NaN)."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


def _signs(rng, n):
    return rng.choice([-1.0, 1.0], n)


def _wide(rng, n, lo, hi):
    return _signs(rng, n) * np.exp2(rng.uniform(lo, hi, n))


def _blocks(layout, hidden_layers):
    """(start, rows, columns) of every network matrix."""
    out, o = [], 0
    for m in range(hidden_layers + 1):
        rows, cols = (16 if m == hidden_layers else 64), (layout.n_inputs if m == 0 else 64)
        out.append((o, rows, cols))
        o += rows * cols
    return out


def _params(kind, h, rng):
    H, n_net, n = h.cfg.network.n_hidden_layers, h.layout.n_network_params, h.layout.n_params
    p = np.empty(n, np.float64)
    table = slice(n_net, n)
    if kind == "wide":  # exponents over the whole FP16 range, weights and features
        p[:n_net] = _wide(rng, n_net, -14, 1)
        p[table] = _wide(rng, n - n_net, -14, 4)
    elif kind == "cancelling":  # neighbouring columns cancel to their last bits
        p[table] = np.repeat(rng.uniform(0.5, 1.0, (n - n_net) // 2), 2)
        for o, r, c in _blocks(h.layout, H):
            w = rng.uniform(0.25, 1.0, (r, c // 2)) * _signs(rng, (r, c // 2))
            p[o:o + r * c] = np.stack([w, -w * (1.0 + np.exp2(rng.integers(-11, -8, w.shape)))], 2).ravel()
    elif kind == "far_cancelling":  # large terms that cancel across a row around small ones
        p[table] = rng.uniform(0.5, 1.0, n - n_net)
        for o, r, c in _blocks(h.layout, H):
            w = rng.uniform(-1.0, 1.0, (r, c)) * 2.0 ** -9
            k = rng.integers(0, c // 2, r)
            big = np.exp2(rng.integers(0, 5, r))
            w[np.arange(r), k], w[np.arange(r), c // 2 + k] = big, -big
            p[o:o + r * c] = w.ravel()
    elif kind in ("limit", "overflow"):  # hidden activations around 65,504, or far beyond it
        p[:n_net] = rng.uniform(-1.0, 1.0, n_net) * 0.25
        p[table] = rng.uniform(-1.0, 1.0, n - n_net) * (3.0e4 if kind == "limit" else 6.5e4)
        if kind == "overflow":
            p[:n_net] *= 16.0
    elif kind == "subnormal":  # products and activations below 2^-14
        p[:n_net] = rng.uniform(-1.0, 1.0, n_net) * 2.0 ** -3
        p[table] = rng.uniform(-1.0, 1.0, n - n_net) * 2.0 ** -12
        o, r, c = _blocks(h.layout, H)[-1]
        p[o:o + r * c] *= 2.0 ** 14
    else:  # saturated outputs
        p[:n_net] = rng.uniform(-1.0, 1.0, n_net) * 0.5
        p[table] = rng.uniform(-1.0, 1.0, n - n_net) * 4.0
        o, r, c = _blocks(h.layout, H)[-1]
        p[o:o + r * c] *= 64.0
    return p.astype(np.float32)


KINDS = ["wide", "cancelling", "far_cancelling", "limit", "overflow", "subnormal", "saturated"]


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("kind", KINDS)
def test_tensor_core_paths_agree(built, kind, precision):
    cfg = nb.default_config(**{"hashgrid.base_resolution": 8, "hashgrid.log2_hashmap_size": 14,
                               "network.precision": precision, "output.primary_visibility_threshold": -1.0,
                               "output.secondary_visibility_threshold": 0.5})
    h, s = handle(cfg, kind="soup64k", seed=2, depth=12)
    with h:
        n = 160003
        rays = torch.from_numpy(scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=6, scaling=1.0)).cuda()
        for seed in (1, 2):
            h.set_params(_params(kind, h, np.random.default_rng(seed)))
            for depth in (1, 2):
                whole = h.query_closest_neural(rays, depth)
                if depth == 1 and kind != "overflow":
                    assert int((whole[:, 8] & 1).sum()) > n // 4
                for a in range(0, n, 1 << 14):
                    part = h.query_closest_neural(rays[a:a + (1 << 14)].contiguous(), depth)
                    assert torch.equal(part, whole[a:a + (1 << 14)]), (seed, depth, a)
