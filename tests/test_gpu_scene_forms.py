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
