"""The cell copy of the coarse grid levels when a query builds it while the parameters are being written:
a scene's query does not hold its models' locks. What it answers meanwhile may be from either state;
once the writing call is over every query follows the new parameters."""

import threading
import time

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_copy_built_during_training_is_dropped(built):
    cfg = nb.default_config(batch_size=1 << 16, **{"hashgrid.log2_hashmap_size": 15})
    h, s = handle(cfg, kind="sphere4k", seed=1)
    n = 1 << 20
    rays = torch.from_numpy(scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
    with h:
        rng = np.random.default_rng(7)
        p = h.params()
        nn = h.layout.n_network_params
        p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
        h.set_params(p)
        scene = nb.Scene()
        scene.add_instance(h)
        scene.query_closest(rays[:1024])  # the scene's buffers
        steps = 1500
        h.run_optimisation(2)
        trainer = threading.Thread(target=h.run_optimisation, args=(steps,))
        trainer.start()
        time.sleep(0.05)
        during = 0
        while trainer.is_alive():  # some of these build the copy in the middle of the training
            scene.query_closest(rays)
            during += 1
        trainer.join()
        assert during >= 3
        torch.cuda.synchronize()
        got = [h.query_closest_neural(rays) for _ in range(3)]
        placed = scene.query_closest(rays)
        scene.close()
        with nb.NBVH(h.cfg) as f:
            f.set_mesh(s["v"], s["f"])
            f.build_classic()
            f.build_neural_cut()
            f.set_params(h.params())
            ref = f.query_closest_neural(rays)
            again = nb.Scene()
            again.add_instance(f)
            placed_ref = again.query_closest(rays)
            again.close()
        for g in got:
            assert torch.equal(g, ref)
        assert torch.equal(placed, placed_ref)
