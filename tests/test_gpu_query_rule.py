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


def _shapes(call, tmp_path, kernel):
    """(grid, block) of the launches of `kernel` during the call."""
    import json
    import torch
    call()
    for _ in range(3):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            call()
            torch.cuda.synchronize()
        p.export_chrome_trace(str(tmp_path / "trace.json"))
        with open(tmp_path / "trace.json") as f:
            events = json.load(f)["traceEvents"]
        found = [(e["args"]["grid"][0], e["args"]["block"][0]) for e in events
                 if kernel in e.get("name", "") and "grid" in e.get("args", {})]
        if found:
            return found
    pytest.skip("no activity records")


def test_launch_shape_of_packet_queries(gpu, bvh, tmp_path):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    scene = gpu.Scene(bvh)
    o, d = scenes.random_rays(300000, seed=1)
    t, tri = scene.intersect_nearest(o, d)
    for blocks in (4, 10):
        scene.set_query_launch(blocks)
        shapes = _shapes(lambda: scene.intersect_nearest(o, d), tmp_path, "k_intersect_packets")
        assert shapes == [(blocks * sms, 128)], shapes
        t2, tri2 = scene.intersect_nearest(o, d)
        assert (tri == tri2).all() and (t.view(np.uint32) == t2.view(np.uint32)).all()


@pytest.mark.parametrize("block", [32, 64, 96, 128])
def test_block_size_of_packet_frames(gpu, bvh, tmp_path, block):
    scene = gpu.Scene(bvh)
    scenes.default_camera(scene.camera)
    w, h = 333, 181
    ref = gpu.Renderer(scene, w, h, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_PACKET).render_frame_u8(3)
    r = gpu.Renderer(scene, w, h, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_PACKET, block_size=block)
    out = r.render_frame_u8(3)
    assert (out[0] == ref[0]).all() and (out[1] == ref[1]).all()
    shapes = _shapes(lambda: r.render_frame_u8(3), tmp_path, "k_render_packets")
    assert [b for _, b in shapes] == [block], shapes


def test_autotuner_times_each_launch_once(gpu):
    from convector_gb300 import autotune
    for order in (gpu.RNG_PATCH, gpu.RNG_GROUP):
        packets = [c for c in autotune.candidates(order) if c["traversal"] == gpu.TRAVERSE_PACKET and "block_size" in c]
        assert len(packets) == (1 if order == gpu.RNG_PATCH else 2)
