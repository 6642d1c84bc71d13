"""The launches that nbvh_last_kernel_time reports for calls that take their rays or rows in an order of
their own from some size on."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_classic_queries(built):
    h, s = handle(kind="sphere4k", seed=1)
    with h:
        rays = torch.from_numpy(scenes.uniform_rays(1 << 19, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
        for query in (h.query_closest_classic, h.query_any_classic):
            query(rays)
            assert h.last_kernel_time()[1] == 3  # bins, placement, traversal
            query(rays[:-1])
            assert h.last_kernel_time()[1] == 1


# below and from the size on whose rows are encoded in place order; a loss scale that is no power of two is
# divided out in a pass of its own
@pytest.mark.parametrize("n,scale,launches", [(4096, 128.0, 4), (4096, 100.0, 5), (196608, 128.0, 6), (196607, 128.0, 4)])
def test_gradients(built, n, scale, launches):
    h, s = handle(nb.default_config(batch_size=4096, **{"optimizer.loss_scale": scale}), kind="sphere4k", seed=1)
    with h:
        rng = np.random.default_rng(3)
        pos = torch.from_numpy(rng.uniform(0, 1, (n, 12)).astype(np.float32)).cuda()
        tgt = torch.from_numpy(rng.uniform(0, 1, (n, 8)).astype(np.float32)).cuda()
        h.run_optimisation(1)  # the call's time is measured there, not by gradients alone
        h.compute_gradients(pos, tgt)
        assert h.last_kernel_time()[1] == launches


@pytest.mark.parametrize("batch,per_step", [(1 << 12, 7), (1 << 18, 9)])
def test_training_steps(built, batch, per_step):
    h, s = handle(nb.default_config(batch_size=batch), kind="sphere4k", seed=1)
    with h:
        h.run_optimisation(3)
        assert h.last_kernel_time()[1] == 3 * per_step
