"""The cell copy of the coarse grid levels follows the parameters: a query after any call that changes
them answers as a new handle with the same parameters does, word for word, whatever copy the query
before it left behind. (The encoder's values from the copy against the table are in test_gpu_tail:
small batches read the table alone, large ones both.)"""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import scenes

pytestmark = pytest.mark.gpu

N = 1 << 20  # the copy is built for the second query of this size


def _params(h, seed):
    rng = np.random.default_rng(seed)
    p = h.params()
    nn = h.layout.n_network_params
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    return p


def _adam(h, stream=None):
    g = torch.rand(h.layout.n_params, device="cuda", generator=torch.Generator("cuda").manual_seed(3)) - 0.5
    torch.cuda.synchronize()
    h.adam_step(g, stream)
    return g


def _adam_other_stream(h, tmp):
    return _adam(h, torch.cuda.Stream())  # the query below runs on the current stream, unordered with it


def _adam_captured(h, tmp):
    g = _adam(h)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        h.adam_step(g)
    yield
    graph.replay()
    torch.cuda.synchronize()


def _load(h, tmp):
    other = nb.NBVH(h.cfg)
    with other:
        other.set_mesh(*h._keep[:2])
        other.build_classic()
        other.build_neural_cut()
        other.set_params(_params(other, 9))
        other.save(str(tmp / "m.bin"))
    h.load(str(tmp / "m.bin"))


WRITERS = {
    "set_params": lambda h, tmp: h.set_params(_params(h, 8)),
    "adam_step": lambda h, tmp: _adam(h),
    "adam_step_other_stream": _adam_other_stream,
    "adam_step_captured": _adam_captured,
    "run_optimisation": lambda h, tmp: h.run_optimisation(2),
    "load": _load,
}


@pytest.mark.parametrize("features", [2, 4])
@pytest.mark.parametrize("writer", sorted(WRITERS))
def test_queries_follow_the_parameters(built, tmp_path, writer, features):
    cfg = nb.default_config(batch_size=1 << 12, **{"hashgrid.n_features_per_level": features,
                                                   "hashgrid.n_levels": 32 // features,
                                                   "hashgrid.log2_hashmap_size": 15})
    h, s = handle(cfg, kind="sphere4k", seed=1)
    with h:
        h.set_params(_params(h, 7))
        rays = torch.from_numpy(scenes.uniform_rays(N, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
        for _ in range(2):
            first = h.query_closest_neural(rays)
        change = WRITERS[writer](h, tmp_path)
        if hasattr(change, "__next__"):  # a captured step: a query between capture and replay
            next(change)
            for _ in range(2):
                h.query_closest_neural(rays)
            next(change, None)
        got, again = h.query_closest_neural(rays), h.query_closest_neural(rays)
        assert torch.equal(again, got)
        torch.cuda.synchronize()
        assert not torch.equal(got, first)
        small = torch.cat([h.query_closest_neural(r) for r in rays[:1 << 15].split(1 << 14)])
        assert torch.equal(small, got[:1 << 15])
        with nb.NBVH(h.cfg) as f:
            f.set_mesh(s["v"], s["f"])
            f.build_classic()
            f.build_neural_cut()
            f.set_params(h.params())
            assert torch.equal(f.query_closest_neural(rays), got)
