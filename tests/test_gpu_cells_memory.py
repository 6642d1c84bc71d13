"""When the cell copy of the coarse grid levels takes memory: only where a kernel reads it, again after an
allocation that failed, no longer once it is given up, and no more than the caller allows."""

import ctypes as C

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

N = 1 << 20  # the second query of this size builds the copy


def _allocations():
    n = C.c_uint64(0)
    assert nb.load_library().nbvh_debug_alloc_count(C.byref(n)) == abi.NBVH_OK
    return n.value


def _model(levels=16, features=2):
    cfg = nb.default_config(batch_size=1 << 12, **{"hashgrid.n_levels": levels, "hashgrid.n_features_per_level": features,
                                                   "hashgrid.log2_hashmap_size": 15})
    h, s = handle(cfg, kind="sphere4k", seed=1)
    rng = np.random.default_rng(7)
    p = h.params()
    nn = h.layout.n_network_params
    p[nn:] = rng.uniform(-0.5, 0.5, p.size - nn).astype(np.float32)
    h.set_params(p)
    rays = torch.from_numpy(scenes.uniform_rays(N, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
    return h, rays


def test_copy_is_one_allocation(built):
    h, rays = _model()
    with h:
        h.query_closest_neural(rays)
        before = _allocations()
        h.query_closest_neural(rays)
        assert _allocations() == before + 1
        h.query_closest_neural(rays)
        assert _allocations() == before + 1


def test_no_copy_where_no_kernel_reads_it(built):
    """A 2-feature grid whose levels are no multiple of the four that its encoder stores at once; a
    handle answered by the classic BLAS."""
    h, rays = _model(levels=6)
    with h:
        h.query_closest_neural(rays)
        before = _allocations()
        for _ in range(3):
            h.query_closest_neural(rays)
        assert _allocations() == before
    h, rays = _model()
    with h:
        h.set_ignore_neural_blas(True)
        h.query_closest_neural(rays)
        before = _allocations()
        for _ in range(3):
            h.query_closest_neural(rays)
        assert _allocations() == before


def test_failed_allocation_is_tried_again(built):
    h, rays = _model()
    lib = nb.load_library()
    with h:
        first = h.query_closest_neural(rays)
        assert lib.nbvh_debug_fail_allocations(0) == abi.NBVH_OK
        try:
            assert torch.equal(h.query_closest_neural(rays), first)  # the table alone
        finally:
            lib.nbvh_debug_fail_allocations(-1)
        before = _allocations()
        for _ in range(3):
            assert torch.equal(h.query_closest_neural(rays), first)
        assert _allocations() == before + 1


def test_copy_given_up_is_freed(built):
    """An Adam step captured into a graph: its replays change the parameters unseen."""
    h, rays = _model()
    with h:
        for _ in range(2):
            h.query_closest_neural(rays)
        g = torch.zeros(h.layout.n_params, device="cuda")
        h.adam_step(g)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            h.adam_step(g)
        free = torch.cuda.mem_get_info()[0]
        h.query_closest_neural(rays)
        assert torch.cuda.mem_get_info()[0] > free
        before = _allocations()
        for _ in range(3):
            h.query_closest_neural(rays)
        assert _allocations() == before


def test_caller_sets_the_size(built):
    h, rays = _model()
    with h:
        h.set_cell_copy(0)
        h.query_closest_neural(rays)
        before = _allocations()
        ref = h.query_closest_neural(rays)
        for _ in range(3):
            assert torch.equal(h.query_closest_neural(rays), ref)
        assert _allocations() == before
        free = torch.cuda.mem_get_info()[0]
        taken = []
        for limit in (16 << 20, 192 << 20, 1 << 40, 1 << 10, 192 << 20, 0):
            h.set_cell_copy(limit)
            for _ in range(3):
                assert torch.equal(h.query_closest_neural(rays), ref)
            taken.append(free - torch.cuda.mem_get_info()[0])
        small, full, more, none, again, off = taken
        assert 0 < small <= 18 << 20 and small < full <= 194 << 20 and more == again == full and none == off == 0
