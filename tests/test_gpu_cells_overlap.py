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


def _model(n):
    cfg = nb.default_config(batch_size=1 << 16, **{"hashgrid.log2_hashmap_size": 15})
    h, s = handle(cfg, kind="sphere4k", seed=1)
    rng = np.random.default_rng(7)
    p = h.params()
    nn = h.layout.n_network_params
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    h.set_params(p)
    return h, s, torch.from_numpy(scenes.uniform_rays(n, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()


def test_copy_waits_for_an_adam_step_on_another_stream(built):
    """The step is still behind other work on its stream when a query of 2^21 rays on this one finds the copy
    due: the build waits for it, and so does the query after the build."""
    h, s, rays = _model(1 << 21)
    with h:
        g = torch.rand(h.layout.n_params, device="cuda", generator=torch.Generator("cuda").manual_seed(3)) - 0.5
        a = torch.rand((4096, 4096), device="cuda")
        b = a @ a
        before = h.query_closest_neural(rays)
        other = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            for _ in range(40):
                torch.mm(a, a, out=b)
        h.adam_step(g, other)
        pending = not other.query()
        got = h.query_closest_neural(rays)
        assert pending
        torch.cuda.synchronize()
        with nb.NBVH(h.cfg) as f:
            f.set_mesh(s["v"], s["f"])
            f.build_classic()
            f.build_neural_cut()
            f.set_params(h.params())
            f.set_cell_copy(0)
            ref = f.query_closest_neural(rays)
        assert torch.equal(got, ref) and not torch.equal(got, before)


def test_copy_built_during_training_is_dropped(built):
    n = 1 << 20
    h, s, rays = _model(n)
    with h:
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
