"""The shortest wait limit: every phase wait of the tensor-core kernels that does not find its phase
complete runs out at once, the one for the weights' copy among them. Whatever is in flight then is
waited for before the kernel exits; the calls report NBVH_ETIMEOUT (or succeed, where nothing had to be
waited for) and answer as before once the limit is back."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_waits_that_run_out_at_once(built, precision):
    cfg = nb.default_config(batch_size=1 << 12, **{"network.precision": precision})
    h, s = handle(cfg, kind="sphere4k", seed=3)
    with h:
        rng = np.random.default_rng(2)
        p = h.params()
        nn = h.layout.n_network_params
        p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
        h.set_params(p)
        feats = torch.from_numpy(rng.uniform(-0.1, 0.1, (100001, h.layout.n_inputs)).astype(np.float32)).cuda()
        feats = (feats.bfloat16() if precision == 1 else feats.half()).contiguous()
        rays = torch.from_numpy(scenes.uniform_rays(1 << 17, s["bbox"][:3], s["bbox"][3:], seed=5)).cuda()
        pos, tgt, _ = h.generate_training_batch(1, 40001)
        calls = {"mlp": lambda: h.mlp_inference(feats), "query": lambda: h.query_closest_neural(rays),
                 "gradients": lambda: h.compute_gradients(pos, tgt)[0]}
        ref = {k: f() for k, f in calls.items()}
        timeouts = 0
        assert h.lib.nbvh_debug_set_wait_limit(h.h, 1) == abi.NBVH_OK
        try:
            for _ in range(3):
                for f in calls.values():
                    try:
                        f()
                    except nb.NBVHError as e:
                        assert e.status == abi.NBVH_ETIMEOUT, e
                        timeouts += 1
        finally:
            h.lib.nbvh_debug_set_wait_limit(h.h, 0)
        assert timeouts > 0
        for k in ("mlp", "query"):
            assert torch.equal(calls[k](), ref[k]), k
        g = ref["gradients"]  # FP32 atomics in any order: entries of up to 160,004 addends
        assert float((calls["gradients"]() - g).abs().max()) <= 1e-4 * float(g.abs().max())
