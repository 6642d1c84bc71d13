"""A server's captured graphs read the cell copy of the coarse grid levels. Requests answered after the
model's parameters changed between them are the records of a new handle with the same parameters,
word for word, whichever call changed them. The copy is made for batches that read it, within the
server's memory budget."""

import ctypes as C

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

N = 1 << 20  # two requests of this size are enough rays for the copy


def _params(h, seed):
    rng = np.random.default_rng(seed)
    p = h.params()
    nn = h.layout.n_network_params
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    return p


def _gradient(h):
    g = torch.rand(h.layout.n_params, device="cuda", generator=torch.Generator("cuda").manual_seed(3)) - 0.5
    torch.cuda.synchronize()
    return g


def _adam(h):
    h.adam_step(_gradient(h))
    torch.cuda.synchronize()


def _adam_captured(h):
    g = _gradient(h)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        h.adam_step(g)
    graph.replay()
    torch.cuda.synchronize()


WRITERS = {"set_params": lambda h, k: h.set_params(_params(h, 8 + k)), "adam_step": lambda h, k: _adam(h),
           "adam_step_captured": lambda h, k: _adam_captured(h), "run_optimisation": lambda h, k: h.run_optimisation(2)}


@pytest.mark.parametrize("writer", sorted(WRITERS))
def test_requests_follow_the_parameters(built, writer):
    cfg = nb.default_config(batch_size=1 << 12, **{"hashgrid.log2_hashmap_size": 15})
    h, s = handle(cfg, kind="sphere4k", seed=1)
    rays = scenes.uniform_rays(N, s["bbox"][:3], s["bbox"][3:], seed=2)
    with h:
        h.set_params(_params(h, 7))
        srv = nb.Server(n_slots=1, hbm_budget_gb=4, max_batch_rays=N, autotune=False)
        try:
            model = srv.add_model(h)

            def ask():
                hits, res = srv.wait(srv.submit_query(model, rays))
                assert res.status == 0
                return hits.view(np.uint32).copy()

            last = [ask() for _ in range(4)][-1]
            for k in range(2):  # the second time the copy of the first change is there
                WRITERS[writer](h, k)
                got = [ask() for _ in range(4)]
                with nb.NBVH(h.cfg) as f:
                    f.set_mesh(s["v"], s["f"])
                    f.build_classic()
                    f.build_neural_cut()
                    f.set_params(h.params())
                    ref = f.query_closest_neural(torch.from_numpy(rays).cuda()).cpu().numpy().view(np.uint32)
                assert not np.array_equal(ref.ravel(), last.ravel())
                for g in got:
                    assert np.array_equal(g.ravel(), ref.ravel())
                last = got[-1]
            assert srv.stats().graph_replays > 0
        finally:
            srv.close()


def _allocations():
    n = C.c_uint64(0)
    assert nb.load_library().nbvh_debug_alloc_count(C.byref(n)) == abi.NBVH_OK
    return n.value


@pytest.mark.parametrize("rays_per_request,budget_gb,copies", [(1 << 14, 8, 0), (1 << 20, 8, 1), (1 << 20, 2.05, 0)])
def test_copy_for_large_batches_within_the_budget(built, rays_per_request, budget_gb, copies):
    """Two slots of 2^20 rays are counted as 1 GiB each: the copy of some 190 MB fits beside them in 8 GiB and not in
    2.05. Requests of 16,384 rays or fewer never read it, however many there are."""
    h, s = handle(nb.default_config(**{"hashgrid.log2_hashmap_size": 15}), kind="sphere4k", seed=1)
    rays = scenes.uniform_rays(rays_per_request, s["bbox"][:3], s["bbox"][3:], seed=2)
    with h:
        h.set_params(_params(h, 7))
        alone = h.query_closest_neural_host(rays).view(np.uint32).ravel()

        def allocations(cell_bytes):
            h.set_cell_copy(cell_bytes)
            before = _allocations()
            srv = nb.Server(n_slots=2, hbm_budget_gb=budget_gb, max_batch_rays=1 << 20, autotune=False)
            try:
                assert srv.stats().slot_capacity_rays == 1 << 20
                model = srv.add_model(h)
                for _ in range(3 * (1 << 20) // rays_per_request + 2):
                    hits, res = srv.wait(srv.submit_query(model, rays))
                    assert res.status == 0
                    assert np.array_equal(hits.view(np.uint32).ravel(), alone)
                return _allocations() - before
            finally:
                srv.close()

        assert allocations(0) + copies == allocations(192 << 20)
