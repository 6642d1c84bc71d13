"""The tensor-core MLP's input widths: rows copied in 128-, 64- or 32-byte swizzled boxes. Against a plain
PyTorch evaluation (FP64 sums) with the same 16-bit roundings; the sums' order alone differs, which can flip a
rounding (2^-11 of an activation) per layer: far below 4e-3 of outputs in (0, 1)."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [16, 32, 48, 64, 80, 96, 112, 128])
@pytest.mark.parametrize("precision,dtype,tol", [(0, torch.float16, 4e-3), (1, torch.bfloat16, 3.2e-2)])
def test_every_input_width(built, width, precision, dtype, tol):
    cfg = nb.default_config(**{"hashgrid.n_levels": width // 16, "hashgrid.n_features_per_level": 4,
                               "hashgrid.log2_hashmap_size": 12, "module.input_segment_points": 4,
                               "network.precision": precision})
    with nb.NBVH(cfg) as h:
        assert h.layout.n_inputs == width
        rng = np.random.default_rng(width)
        p = h.params()
        nn = h.layout.n_network_params
        p[:nn] = rng.normal(0.0, 0.18, nn).astype(np.float32)
        h.set_params(p)
        n = 5 * 152 * 128 + 77  # several tiles for some groups, a ragged last one
        x = torch.from_numpy(rng.uniform(-1.0, 1.0, (n, width)).astype(np.float32)).cuda().to(dtype)
        got = h.mlp_inference(x)
        w = torch.from_numpy(p[:nn]).cuda().to(dtype).double()
        o, a = 0, x.double()
        for j in range(cfg.network.n_hidden_layers + 1):
            rows, cols = (64 if j < cfg.network.n_hidden_layers else 16), a.shape[1]
            z = a @ w[o:o + rows * cols].view(rows, cols).T
            o += rows * cols
            a = z.clamp(min=0).to(dtype).double() if j < cfg.network.n_hidden_layers else torch.sigmoid(z[:, :8])
        assert o == nn
        assert (got.double() - a).abs().max() <= tol
