"""Which kernels a nearest-hit query runs, by the profiler's activity records, and
that the stack settings give the same hits.
"""

import numpy as np
import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bvh(gpu):
    return gpu.Bvh.build(scenes.spheres_and_boxes(3000, 5, obj=False)[0])


def _kernels(call):
    """Names of what the device ran during the call."""
    import torch
    call()
    torch.cuda.synchronize()
    for _ in range(3):  # (the first profile of a process may come back empty)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            call()
            torch.cuda.synchronize()
        names = [e.name for e in p.events()]
        if names:
            return names
    pytest.skip("no activity records")


@pytest.mark.parametrize("traversal,direct,persistent", [(0, "k_intersect_warp", "k_intersect_packets"),
                                                         (1, "k_intersect_lanes", "k_intersect_refill")])
@pytest.mark.parametrize("stack", [None, 0, 4, 8, 12])
def test_small_queries_are_direct_whatever_the_stack(gpu, bvh, traversal, direct, persistent, stack):
    scene = gpu.Scene(bvh)
    if stack is not None:
        scene.set_query_stack(stack)
    o, d = scenes.random_rays(5000, seed=1)
    names = _kernels(lambda: scene.intersect_nearest(o, d, traversal=traversal))
    assert any(direct in n for n in names) and not any(persistent in n for n in names), names
    # A launch shape selects the persistent kernels: hits and their counter in device memory, copied out.
    scene.set_query_launch(10)
    names = _kernels(lambda: scene.intersect_nearest(o, d, traversal=traversal))
    assert any(persistent in n for n in names) and not any(direct in n for n in names), names
    assert any("Memcpy DtoH" in n for n in names), names


def test_tuned_scene_keeps_its_small_queries(gpu, bvh):
    import torch
    from convector_gb300 import autotune
    scene = gpu.Scene(bvh)
    o, d = scenes.random_rays(300000, seed=2)
    rays = torch.from_numpy(np.ascontiguousarray(np.concatenate([o.T, d.T]))).cuda()
    t, tri = torch.empty(300000, device="cuda"), torch.empty(300000, dtype=torch.int32, device="cuda")
    for name in ("packet8/0", "single/8", "single/8/s0", "single/8/s4", "single/8/s12"):
        autotune.tune_query(scene, rays, t, tri, shapes=[name])
        for traversal, direct in ((0, "k_intersect_warp"), (1, "k_intersect_lanes")):
            names = _kernels(lambda: scene.intersect_nearest(o[:999], d[:999], traversal=traversal))
            assert any(direct in n for n in names), (name, names)


@pytest.mark.parametrize("stack", [0, 4, 8, 12])
@pytest.mark.parametrize("blocks", [0, 8, 10])
def test_stack_settings_agree(gpu, orc, bvh, stack, blocks):
    scene, osc = gpu.Scene(bvh), orc.OracleScene.from_bvh(bvh)
    n = 270001  # beyond the direct kernels
    o, d = scenes.random_rays(n, seed=3)
    scene.set_query_stack(stack)
    scene.set_query_launch(blocks)
    t, tri = scene.intersect_nearest(o, d, traversal=gpu.TRAVERSE_SINGLE)
    ot, otri = osc.intersect(o, d, mode=gpu.TRAVERSE_SINGLE)
    assert (tri == otri).all() and (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("n,traversal,kernel", [(20000, 0, "k_intersect_warp"), (50000, 0, "k_intersect_octets"),
                                                (1 << 20, 0, "k_intersect_packets<6"),
                                                (300000, 1, "k_intersect_refill<8, false, 16, (cvx::Form)1")])
def test_kernels_of_a_scene_without_wide_records(gpu, n, traversal, kernel):
    b = gpu.Bvh.build(scenes.spheres_and_boxes(3000, 5, obj=False)[0])
    f = b.nodes.view(np.float32)
    f[0:2, 0:3] -= np.float32(0.5)
    f[0:2, 3:6] += np.float32(0.5)
    scene = gpu.Scene(b)
    o, d = scenes.random_rays(n, seed=1)
    names = _kernels(lambda: scene.intersect_nearest(o, d, traversal=traversal))
    assert any(kernel in k for k in names), names
