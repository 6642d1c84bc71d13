"""A call whose buffers cannot grow reports NBVH_ENOMEM whichever of its allocations fails, and leaves nothing
half-grown behind: a smaller call that the old buffers held and the same call again answer as before."""

import numpy as np
import pytest
import torch

import nbvh_gb300 as nb
from helpers import handle
from nbvh_gb300 import abi, scenes

pytestmark = pytest.mark.gpu

SMALL, LARGE = 40000, 1 << 19  # the large ones take rays in coherence order and sort their lists


def _calls(s):
    large = torch.from_numpy(scenes.uniform_rays(LARGE, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
    small = large[:SMALL].contiguous()

    def path(h, width, height):
        org, tgt, up = scenes.orbit_camera(s["bbox"][:3], s["bbox"][3:], seed=9)
        cam = nb.render_request(width, height, org, tgt, up, 45.0)
        return h.render_path(nb.path_request(cam, spp=1, max_bounces=1, seed=4))[0]

    return {
        "neural": lambda h, grow: h.query_closest_neural(large if grow else small),
        "classic": lambda h, grow: h.query_closest_classic(large if grow else small),
        "path": lambda h, grow: path(h, 1024, 512) if grow else path(h, 200, 200),
    }


@pytest.mark.parametrize("kind", ["neural", "classic", "path"])
def test_every_failing_allocation(built, kind):
    lib = nb.load_library()
    ref, failures = None, 0
    for after in range(64):
        h, s = handle(kind="sphere4k", seed=1)
        with h:
            call = _calls(s)[kind]
            if ref is None:
                ref = call(h, False).clone(), call(h, True).clone()
                h.close()
                h, _ = handle(kind="sphere4k", seed=1)
            assert torch.equal(call(h, False), ref[0])
            torch.cuda.empty_cache()
            status = abi.NBVH_OK
            assert lib.nbvh_debug_fail_allocations(after) == abi.NBVH_OK
            try:
                call(h, True)
            except nb.NBVHError as e:
                status = e.status
            finally:
                lib.nbvh_debug_fail_allocations(-1)
            if status == abi.NBVH_OK:
                break
            assert status == abi.NBVH_ENOMEM
            failures += 1
            assert torch.equal(call(h, False), ref[0])
            assert torch.equal(call(h, True), ref[1])
            h.close()
    assert status == abi.NBVH_OK and failures >= {"neural": 16, "classic": 3, "path": 16}[kind]


def test_every_failing_allocation_of_a_scene(built):
    lib = nb.load_library()
    h, s = handle(kind="sphere4k", seed=1)
    large = torch.from_numpy(scenes.uniform_rays(LARGE, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
    small = large[:SMALL].contiguous()
    ref, failures = None, 0
    with h:
        for after in range(64):
            scene = nb.Scene()
            scene.add_instance(h)
            if ref is None:
                ref = scene.query_closest(small).clone(), scene.query_closest(large).clone()
                scene.close()
                scene = nb.Scene()
                scene.add_instance(h)
            status = []
            for rays, expect in ((small, ref[0]), (large, ref[1])):
                assert lib.nbvh_debug_fail_allocations(after) == abi.NBVH_OK
                try:
                    scene.query_closest(rays)
                    status.append(abi.NBVH_OK)
                except nb.NBVHError as e:
                    status.append(e.status)
                finally:
                    lib.nbvh_debug_fail_allocations(-1)
                assert torch.equal(scene.query_closest(small), ref[0])
                assert torch.equal(scene.query_closest(rays), expect)
            scene.close()
            assert all(x in (abi.NBVH_OK, abi.NBVH_ENOMEM) for x in status)
            failures += sum(x != abi.NBVH_OK for x in status)
            if not any(status):
                break
    assert not any(status) and failures >= 20


def test_error_is_reported_once(built):
    """A call that fails in the CUDA runtime (no query was timed yet) leaves nothing for the next one's check of
    its launches."""
    h, s = handle(kind="sphere4k", seed=1)
    rays = torch.from_numpy(scenes.uniform_rays(SMALL, s["bbox"][:3], s["bbox"][3:], seed=2)).cuda()
    with h:
        with pytest.raises(nb.NBVHError) as e:
            h.last_kernel_time()
        assert e.value.status == abi.NBVH_EDEVICE
        first = h.query_closest_neural(rays)
        assert torch.equal(h.query_closest_neural(rays), first)
        assert h.last_kernel_time()[0] > 0.0
