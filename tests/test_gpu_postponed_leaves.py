"""Traversal with postponed leaves (RefillRay::walk) against the oracle's
single-ray traversal, bit for bit: scenes whose leaves are large, whose nodes
do not nest (which keep the x86 form), rays that start on box corners and rays
with a short far distance, at counts around a claim's 32 rays.
"""

import numpy as np
import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene_arrays(gpu, kind):
    tris = scenes.spheres_and_boxes(3000, 5, obj=False)[0]
    if kind == "large leaves":  # stacks of coincident triangles: leaves of several triangles
        tris = np.concatenate([np.repeat(tris[:40], 20, axis=0), tris])
    b = gpu.Bvh.build(tris)
    nodes = b.nodes.copy()
    if kind == "not nested":  # every third node reaches out of its parent
        f = nodes.view(np.float32)
        f[2::3, 3:6] += np.float32(0.25)
    return b, nodes


def _rays(nodes, n, seed):
    o, d = scenes.random_rays(n, seed=seed)
    f = nodes.view(np.float32)
    corners = np.stack([f[:, [a, b, c]] for a in (0, 3) for b in (1, 4) for c in (2, 5)], 1).reshape(-1, 3)
    k = n // 2
    o[:k] = corners[np.random.default_rng(seed).integers(0, corners.shape[0], k)]
    return o, d


@pytest.mark.parametrize("kind", ["plain", "large leaves", "not nested"])
@pytest.mark.parametrize("n,far", [(1, 1.0e5), (31, 1.0e5), (33, 1.0e5), (40007, 1.0e5), (40007, 0.5)])
def test_query_equals_oracle(gpu, orc, kind, n, far):
    b, nodes = _scene_arrays(gpu, kind)
    b.nodes = nodes
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, nodes)
    o, d = _rays(nodes, n, seed=n)
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        t, tri = scene.intersect_nearest(o, d, far=far, traversal=traversal)
        ot, otri = osc.intersect(o, d, far=far, mode=traversal)
        assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
        assert (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("kind", ["plain", "large leaves", "not nested"])
@pytest.mark.parametrize("refill", ["REFILL_ALL", "REFILL_NONE"])
def test_frame_equals_oracle(gpu, orc, kind, refill):
    b, nodes = _scene_arrays(gpu, kind)
    b.nodes = nodes
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, nodes)
    # the eye on a box corner of the tree, so that camera rays meet tied zeros
    f = nodes.view(np.float32)
    scenes.default_camera(scene.camera, eye=tuple(float(v) for v in f[4, 3:6]), target=(0.0, 1.0, -2.0))
    r = gpu.Renderer(scene, 83, 45, traversal=gpu.TRAVERSE_SINGLE, refill_mode=getattr(gpu, refill))
    rgba, gb = r.render_frame_u8(9)
    orgba, ogb, ocol, orays = osc.render(scene.camera.as_array(), 83, 45, 9, rng_order=orc.RNG_GROUP, traversal=1)
    assert (rgba == orgba).all() and (gb == ogb).all()
    assert (r.read_frame_f32().view(np.uint32) == ocol.view(np.uint32)).all()
    assert r.stats()[0] == orays
