"""Scenes that keep the pair records, or whose node array holds more than their
tree, against the oracle, bit for bit.
"""

import numpy as np
import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index,length", [(0xFFFFFFFE, 0), (0, 0), (0xFFFFFFFF, 40)])
def test_padding_behind_the_tree(gpu, orc, index, length):
    """Nodes that the roots do not reach, of any contents."""
    b = gpu.Bvh.build(scenes.spheres_and_boxes(600, 5, obj=False)[0])
    osc = orc.OracleScene(b.triangles, b.nodes.copy())
    pad = np.zeros((4, 8), np.uint32)
    pad.view(np.float32)[:, :6] = np.nan
    pad[:, 6:8] = (index, length)
    b.nodes = np.concatenate([b.nodes, pad])
    scene = gpu.Scene(b)
    o, d = scenes.random_rays(2003, seed=1)
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        t, tri = scene.intersect_nearest(o, d, traversal=traversal)
        ot, otri = osc.intersect(o, d, mode=traversal)
        assert (tri == otri).all() and (t.view(np.uint32) == ot.view(np.uint32)).all()


def test_scene_without_room_for_the_wide_records(gpu, orc):
    """The one allocation of scene creation that may fail: the scene then keeps to the pairs."""
    b = gpu.Bvh.build(scenes.spheres_and_boxes(600, 5, obj=False)[0])
    try:
        for k in range(100):
            gpu.inject_allocation_failure(k)
            try:
                scene = gpu.Scene(b)
            except gpu.CvxError as e:
                assert "injected" in str(e)
                continue
            break
        # The failure has happened: the next allocation succeeds.
        w, h = 48, 20
        scenes.default_camera(scene.camera)
        r = gpu.Renderer(scene, w, h, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_SINGLE)
    finally:
        gpu.inject_allocation_failure(-1)
    osc = orc.OracleScene.from_bvh(b)
    rgba, gb = r.render_frame_u8(3)
    orgba, ogb, _, _ = osc.render(scene.camera.as_array(), w, h, 3, rng_order=orc.RNG_GROUP, traversal=1)
    assert (rgba == orgba).all() and (gb == ogb).all()
    o, d = scenes.random_rays(2003, seed=1)
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        t, tri = scene.intersect_nearest(o, d, traversal=traversal)
        ot, otri = osc.intersect(o, d, mode=traversal)
        assert (tri == otri).all() and (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("kind", ["loose", "tight, on box corners"])
def test_packets_in_step_cull_either_child_of_a_pair(gpu, orc, kind):
    """A million packet rays over the pairs: a scene with loose roots, and rays that start on box corners (whose
    packets take pairs for the steps with tied zeros). A pair's first child is culled like its second."""
    b = gpu.Bvh.build(scenes.spheres_and_boxes(3000, 5, obj=False)[0])
    f = b.nodes.view(np.float32)
    n = (1 << 20) + 5
    o, d = scenes.random_rays(n, seed=n)
    if kind == "loose":
        f[0:2, 0:3] -= np.float32(0.5)
        f[0:2, 3:6] += np.float32(0.5)
    else:
        k = np.random.default_rng(1).integers(0, f.shape[0], n // 8 + 1).repeat(8)[:n]
        axis = np.random.default_rng(2).integers(0, 3, n)
        o[np.arange(n), axis] = f[k, axis]
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, b.nodes)
    ot, otri = osc.intersect(o, d, mode=gpu.TRAVERSE_PACKET)
    t, tri = scene.intersect_nearest(o, d, traversal=gpu.TRAVERSE_PACKET)
    assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
    assert (t.view(np.uint32) == ot.view(np.uint32)).all()
