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

def _loose(gpu, big=False):
    """A tree whose roots reach further than their children: the select form, but no wide records."""
    b = gpu.Bvh.build(scenes.spheres_and_boxes(3000, 5, obj=False)[0])
    f = b.nodes.view(np.float32)
    f[0:2, 0:3] -= np.float32(2.0e18 if big else 0.5)
    f[0:2, 3:6] += np.float32(2.0e18 if big else 0.5)
    return b


def _under_a_chain(gpu, levels):
    """A built tree under `levels` pairs of a small triangle's leaf and the rest."""
    b = gpu.Bvh.build(scenes.spheres_and_boxes(3000, 5, obj=False)[0])
    nodes, tris = b.nodes.copy(), b.triangles
    f = nodes.view(np.float32)
    lo, hi = f[:2, 0:3].min(0), f[:2, 3:6].max(0)
    extra = np.zeros((levels, 16), np.uint32)
    at = np.linspace(lo, hi, levels + 2, dtype=np.float32)[1:-1]
    step = np.float32(0.05)
    extra.view(np.float32)[:, 0:9] = np.concatenate([at, at + [step, 0, 0], at + [0, step, step]], 1)
    extra[:, 15] = 0x00FFFFFF
    nodes[nodes[:, 7] == 0, 6] += 2 * levels
    top = np.zeros((2 * levels, 8), np.uint32)
    g = top.view(np.float32)
    for p in range(levels):
        g[2 * p, 0:3], g[2 * p, 3:6] = at[p], at[p] + step
        g[2 * p + 1, 0:3], g[2 * p + 1, 3:6] = lo, hi + step
        top[2 * p, 6:8] = (tris.shape[0] + p, 1)
        top[2 * p + 1, 6:8] = (2 * p + 2, 0)
    b.nodes, b.triangles = np.concatenate([top, nodes]), np.concatenate([tris, extra])
    return b


@pytest.mark.parametrize("make", [_loose, lambda gpu: _loose(gpu, True), lambda gpu: _under_a_chain(gpu, 75)],
                         ids=["loose", "large bounds", "deep"])
@pytest.mark.parametrize("n", [32768, 32769, 262145, (1 << 20) - 1, (1 << 20) + 5])
def test_queries_without_wide_records(gpu, orc, make, n):
    """Both sides of the limits between one packet per warp, a packet per octet and packets in step."""
    b = make(gpu)
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, b.nodes)
    o, d = scenes.random_rays(n, seed=n)
    o[::97] = b.nodes.view(np.float32)[-1, 0:3]  # on a box corner
    d[1::97] = [0.0, 0.0, -1.0]                  # beyond the select form
    o[2::97, 1] = np.float32(3.0e19)             # an origin beyond the wide records' bound
    for traversal in (gpu.TRAVERSE_PACKET, gpu.TRAVERSE_SINGLE):
        ot, otri = osc.intersect(o, d, mode=traversal)
        for blocks_per_sm in (0, 8):
            scene.set_query_launch(blocks_per_sm)
            t, tri = scene.intersect_nearest(o, d, traversal=traversal)
            assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
            assert (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("make", [_loose, lambda gpu: _loose(gpu, True), lambda gpu: _under_a_chain(gpu, 40),
                                  lambda gpu: _under_a_chain(gpu, 75)],
                         ids=["loose", "large bounds", "chain of 40", "chain of 75"])
@pytest.mark.parametrize("form", ["packets", "REFILL_ALL", "REFILL_NONE"])
@pytest.mark.parametrize("w,h", [(83, 45), (1000, 605)])
def test_frames_without_wide_records(gpu, orc, make, form, w, h):
    """Shallow and deep trees, and frames on both sides of the packets' limit."""
    b = make(gpu)
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, b.nodes)
    scenes.default_camera(scene.camera)
    packets = form == "packets"
    r = gpu.Renderer(scene, w, h, rng_order=gpu.RNG_GROUP,
                     traversal=gpu.TRAVERSE_PACKET if packets else gpu.TRAVERSE_SINGLE,
                     refill_mode=gpu.REFILL_AFTER_CAMERA if packets else getattr(gpu, form))
    rgba, gb = r.render_frame_u8(9)
    orgba, ogb, ocol, orays = osc.render(scene.camera.as_array(), w, h, 9, rng_order=orc.RNG_GROUP,
                                         traversal=int(not packets))
    assert (rgba == orgba).all() and (gb == ogb).all()
    assert (r.read_frame_f32().view(np.uint32) == ocol.view(np.uint32)).all()
    assert r.stats()[0] == orays


@pytest.mark.parametrize("make", [_loose, lambda gpu: _under_a_chain(gpu, 75)], ids=["loose", "deep"])
def test_samples_and_waves_without_wide_records(gpu, make):
    """Several samples in one launch, and waves of such scenes alone and with one that has the records,
    equal frame after frame."""
    scs = [gpu.Scene(make(gpu)), gpu.Scene(gpu.Bvh.build(scenes.spheres_and_boxes(600, 5, obj=False)[0]))]
    w, h, spp = 83, 45, 3
    cam = scenes.default_camera(gpu.Camera())
    alone = []
    for s in scs:
        r = gpu.Renderer(s, w, h, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_SINGLE, refill_mode=gpu.REFILL_NONE)
        r.set_camera(cam)
        for i in range(spp):
            r.accumulate_frame_f32(5 + i)
        alone.append((r.read_accumulator(), r.resolve_u8(spp)))
    r = gpu.Renderer(scs[0], w, h, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_SINGLE)
    r.set_camera(cam)
    r.accumulate_frames_f32(5, spp)
    assert (r.read_accumulator().view(np.uint32) == alone[0][0].view(np.uint32)).all()
    for graph in (0, 1):
        batch = gpu.Batch(scs, max_groups=1 << 14, max_pixels=3 * w * h, mode=gpu.MODE_MEGAKERNEL,
                          refill_mode=gpu.REFILL_ALL, use_graph=graph)
        for which in ([0, 0], [0, 1], [1, 1], [0, 0]):
            imgs = batch.render([gpu.View(k, w, h, spp, 5, cam) for k in which])[0]
            assert all((img == alone[k][1]).all() for k, img in zip(which, imgs))
        server = gpu.Server(scs, framebuffer_bytes=1 << 24, max_groups=1 << 14, kernel_mode=1, samples_per_wave=2,
                            refill_mode=gpu.REFILL_ALL, use_graph=graph)
        ids = [server.submit(k, w, h, spp, cam, frame_base=5) for k in (0, 1, 0)]
        for rid, k in zip(ids, (0, 1, 0)):
            st, img, _ = server.wait(rid)
            assert st == 0 and (img == alone[k][1]).all()
        server.close()
