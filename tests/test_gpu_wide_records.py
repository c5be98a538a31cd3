"""Traversal over the wide records with postponed leaves (RefillRay::walk)
against the oracle's traversals, bit for bit: scenes whose leaves are large,
whose nodes do not nest or enclose loosely, whose tree is too deep, or whose
bounds are too large (which keep the x86 form), rays that start on box corners
(tied zeros in the slab test), directions beyond the select form, and rays with
a short far distance, at counts around a claim's 32 rays.
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
    if kind == "loose":  # the roots reach further than their children
        f = nodes.view(np.float32)
        f[0:2, 0:3] -= np.float32(0.5)
        f[0:2, 3:6] += np.float32(0.5)
    return b, nodes


def _chain(n):
    """A chain of n pairs, each node 0 a leaf and node 1 the rest: n + 1 levels deep."""
    tris = np.zeros((n + 1, 16), np.uint32)
    f = tris.view(np.float32)
    x = np.arange(n + 1, dtype=np.float32) * np.float32(0.02) - np.float32(1.0)
    f[:, 0:9] = np.stack([x, x * 0 + 0.5, x * 0 - 2, x, x * 0 + 1.5, x * 0 - 2.5, x, x * 0 + 1, x * 0 - 1], 1)
    tris[:, 15] = 0x00FFFFFF
    tris[::4, 15] |= 0x40000000
    nodes = np.zeros((2 * n, 8), np.uint32)
    g = nodes.view(np.float32)
    lo, hi = np.array([0.5, -2.5], np.float32), np.array([1.5, -1.0], np.float32)
    for p in range(n):
        for k, (a, b) in enumerate(((p, p), (p + 1, n))):
            g[2 * p + k, 0:6] = [x[a], lo[0], lo[1], x[b], hi[0], hi[1]]
        nodes[2 * p, 6:8] = (p, 1)
        nodes[2 * p + 1, 6:8] = (2 * p + 2, 0) if p + 1 < n else (n, 1)
    return tris, nodes


def _rays(nodes, n, seed):
    o, d = scenes.random_rays(n, seed=seed)
    f = nodes.view(np.float32)
    corners = np.stack([f[:, [a, b, c]] for a in (0, 3) for b in (1, 4) for c in (2, 5)], 1).reshape(-1, 3)
    k = n // 2
    o[:k] = corners[np.random.default_rng(seed).integers(0, corners.shape[0], k)]
    return o, d


@pytest.mark.parametrize("kind", ["plain", "large leaves", "not nested", "loose"])
@pytest.mark.parametrize("n,far", [(1, 1.0e5), (31, 1.0e5), (33, 1.0e5), (40007, 1.0e5), (40007, 0.5)])
def test_query_equals_oracle(gpu, orc, kind, n, far):
    b, nodes = _scene_arrays(gpu, kind)
    b.nodes = nodes
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, nodes)
    o, d = _rays(nodes, n, seed=n)
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        ot, otri = osc.intersect(o, d, far=far, mode=traversal)
        for blocks_per_sm in (0, 8):  # the small-query kernels, the persistent ones
            scene.set_query_launch(blocks_per_sm)
            t, tri = scene.intersect_nearest(o, d, far=far, traversal=traversal)
            assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
            assert (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("kind", ["plain", "large leaves", "not nested", "loose"])
@pytest.mark.parametrize("form", ["REFILL_ALL", "REFILL_NONE", "packets", "patches"])
@pytest.mark.parametrize("w,h", [(83, 45), (1, 1), (17, 5)])
def test_frame_equals_oracle(gpu, orc, kind, form, w, h):
    b, nodes = _scene_arrays(gpu, kind)
    b.nodes = nodes
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, nodes)
    # the eye on a box corner of the tree, so that camera rays meet tied zeros
    f = nodes.view(np.float32)
    scenes.default_camera(scene.camera, eye=tuple(float(v) for v in f[4, 3:6]), target=(0.0, 1.0, -2.0))
    single = form.startswith("REFILL")
    order = "RNG_PATCH" if form == "patches" else "RNG_GROUP"
    r = gpu.Renderer(scene, w, h, rng_order=getattr(gpu, order), traversal=gpu.TRAVERSE_SINGLE if single else gpu.TRAVERSE_PACKET,
                     refill_mode=getattr(gpu, form) if single else gpu.REFILL_AFTER_CAMERA)
    rgba, gb = r.render_frame_u8(9)
    orgba, ogb, ocol, orays = osc.render(scene.camera.as_array(), w, h, 9, rng_order=getattr(orc, order),
                                         traversal=int(single))
    assert (rgba == orgba).all() and (gb == ogb).all()
    assert (r.read_frame_f32().view(np.uint32) == ocol.view(np.uint32)).all()
    assert r.stats()[0] == orays


@pytest.mark.parametrize("pairs", [1, 2, 79, 80, 81, 125])
def test_chains_equal_oracle(gpu, orc, pairs):
    """Trees of 2 levels (every child a leaf) up to the deepest accepted, on both
    sides of the deepest with wide records (80 levels)."""
    tris, nodes = _chain(pairs)
    b = type("B", (), {"triangles": tris, "nodes": nodes})()
    scene, osc = gpu.Scene(b), orc.OracleScene(tris, nodes)
    o, d = _rays(nodes, 2003, seed=pairs)
    d[::5] = [1.0, 0.0, 0.0]                 # axis-parallel, through every level
    d[1::5] *= np.float32(1.0e-30)           # reciprocals beyond the select form
    d[2::5] *= np.float32(3.0)
    o[3::5] = o[3::5] * np.float32(1.0e25)   # origins beyond it
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        ot, otri = osc.intersect(o, d, mode=traversal)
        for blocks_per_sm in (0, 8):
            scene.set_query_launch(blocks_per_sm)
            t, tri = scene.intersect_nearest(o, d, traversal=traversal)
            assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
            assert (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("scale", [1.0e-4, 1.0, 1.0e16, 1.0e18])
def test_scales_equal_oracle(gpu, orc, scale):
    """Scenes whose distances underflow the zero check or whose bounds exceed the select form's."""
    tris = scenes.spheres_and_boxes(600, 5, obj=False)[0].copy()
    tris.view(np.float32)[:, :9] *= np.float32(scale)
    b = gpu.Bvh.build(tris)
    scene, osc = gpu.Scene(b), orc.OracleScene.from_bvh(b)
    o, d = scenes.random_rays(3001, seed=3)
    o = (o * np.float32(scale)).astype(np.float32)
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        t, tri = scene.intersect_nearest(o, d, far=1.0e30, traversal=traversal)
        ot, otri = osc.intersect(o, d, far=1.0e30, mode=traversal)
        assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
        assert (t.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("width", [16, 48, 64])
def test_patch_widths_equal_oracle(gpu, orc, width):
    """Patches of other widths, on a view whose groups end after any number of
    bounces (what a round guesses from the groups before is then often wrong)."""
    b, nodes = _scene_arrays(gpu, "plain")
    scene, osc = gpu.Scene(b), orc.OracleScene(b.triangles, nodes)
    scenes.default_camera(scene.camera)
    w, h = 150, 70
    origins = [(0, 0), (64, 4), (144, 60), (96, 12)]
    r = gpu.Renderer(scene, w, h)
    rgba, gb = np.full((h, w), 7, np.uint32), np.full((h, w), 7, np.uint32)
    r.render_patches_u8(width, origins, 5, rgba, gb)
    orgba, ogb = np.full((h, w), 7, np.uint32), np.full((h, w), 7, np.uint32)
    orays = osc.render_patches(scene.camera.as_array(), w, h, 5, width, origins, traversal=0, rgba=orgba, gbuf=ogb)
    assert (rgba == orgba).all() and (gb == ogb).all()
    assert r.stats()[0] == orays


@pytest.mark.parametrize("n", [131071, 131072, 131073, 262143, 262144, 262145])
def test_query_forms_agree_at_their_limits(gpu, n):
    """Host and device queries on both sides of the direct forms' limits equal the copying, persistent one."""
    import torch
    b, _ = _scene_arrays(gpu, "plain")
    scene = gpu.Scene(b)
    o, d = scenes.random_rays(n, seed=n)
    rays = torch.from_numpy(np.ascontiguousarray(np.concatenate([o.T, d.T]))).cuda()
    t = torch.empty(n, dtype=torch.float32, device="cuda")
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    for traversal in (gpu.TRAVERSE_SINGLE, gpu.TRAVERSE_PACKET):
        scene.set_query_launch(8)
        scene.set_host_access(gpu.HOST_ACCESS_COPY)
        ot, otri = scene.intersect_nearest(o, d, traversal=traversal)
        scene.set_query_launch(0)
        scene.set_host_access(gpu.HOST_ACCESS_AUTO)
        ht, htri = scene.intersect_nearest(o, d, traversal=traversal)
        scene.intersect_nearest_device(rays, t, tri, traversal=traversal)
        torch.cuda.synchronize()
        for a, c in ((ht, htri), (t.cpu().numpy(), tri.cpu().numpy())):
            assert (c == otri).all() and (a.view(np.uint32) == ot.view(np.uint32)).all()


@pytest.mark.parametrize("shift", [0, 5])
def test_small_query_may_overwrite_its_rays(gpu, shift):
    """Hits written over the ray columns, exactly or shifted, as any buffers of the C call may be."""
    b, _ = _scene_arrays(gpu, "plain")
    scene = gpu.Scene(b)
    n = 3001
    o, d = scenes.random_rays(n, seed=1)
    t, tri = scene.intersect_nearest(o, d)
    cols = [np.ascontiguousarray(a[:, k]) for a in (o, d) for k in range(3)]
    buf = np.zeros(n + shift, np.float32)
    buf[:n] = cols[0]
    out_t, out_tri = buf[shift:], cols[4].view(np.int32)
    ptr = [gpu._ptr(buf[:n])] + [gpu._ptr(c) for c in cols[1:]]
    gpu._check(gpu.lib().cvx_intersect_nearest(scene._h, *ptr, n, 1.0e5, gpu.TRAVERSE_PACKET, gpu._ptr(out_t),
                                               gpu._ptr(out_tri)))
    assert (out_tri == tri).all() and (out_t.view(np.uint32) == t.view(np.uint32)).all()


@pytest.mark.parametrize("most", [2, 3, 7, 8, 31, 70])
def test_pooled_leaves_equal_oracle(gpu, orc, most):
    """Trees deeper than 40 levels, whose leaves' triangles are spread over the warp: leaves of 1 to `most`
    triangles, each one twice (ties), on both sides of a pass's seven per lane and 32 per warp."""
    pairs = 60
    rng = np.random.default_rng(most)
    tris, nodes = _chain(pairs)
    lens = rng.integers(1, most + 1, pairs + 1)
    lens[::7] = most
    first = np.concatenate([[0], np.cumsum(lens)])
    tris = np.repeat(tris, lens, axis=0)
    f = tris.view(np.float32)
    shift = np.repeat(rng.uniform(-0.4, 0.4, (f.shape[0] + 1) // 2).astype(np.float32), 2)[: f.shape[0]]
    f[:, [1, 4, 7]] += shift[:, None] * np.float32(0.5)
    for p in range(pairs):
        nodes[2 * p, 6:8] = (first[p], lens[p])
    nodes[2 * pairs - 1, 6:8] = (first[pairs], lens[pairs])
    g = nodes.view(np.float32)
    g[:, 1], g[:, 4] = 0.25, 1.75
    b = type("B", (), {"triangles": tris, "nodes": nodes})()
    scene, osc = gpu.Scene(b), orc.OracleScene(tris, nodes)
    o, d = _rays(nodes, 5003, seed=most)
    d[::2] = d[::2] * np.float32([1.0, 0.1, 0.1])  # through many levels
    t, tri = (scene.set_query_launch(8), scene.intersect_nearest(o, d, traversal=gpu.TRAVERSE_SINGLE))[1]
    ot, otri = osc.intersect(o, d, mode=gpu.TRAVERSE_SINGLE)
    assert (tri == otri).all(), np.nonzero(tri != otri)[0][:10]
    assert (t.view(np.uint32) == ot.view(np.uint32)).all()
    # frames, and a wave of two scenes
    w, h = 83, 45
    cam = scenes.default_camera(gpu.Camera(), eye=(-0.9, 1.0, 0.2), target=(0.0, 1.0, -2.0))
    scenes.default_camera(scene.camera, eye=(-0.9, 1.0, 0.2), target=(0.0, 1.0, -2.0))
    orgba, ogb, ocol, orays = osc.render(cam.as_array(), w, h, 9, rng_order=orc.RNG_GROUP, traversal=1)
    r = gpu.Renderer(scene, w, h, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_SINGLE, refill_mode=gpu.REFILL_ALL)
    rgba, gb = r.render_frame_u8(9)
    assert (rgba == orgba).all() and (gb == ogb).all() and r.stats()[0] == orays
    other = gpu.Scene(gpu.Bvh.build(scenes.spheres_and_boxes(600, 5, obj=False)[0]))
    batch = gpu.Batch([other, scene], max_groups=1 << 14, max_pixels=3 * w * h, mode=gpu.MODE_MEGAKERNEL,
                      refill_mode=gpu.REFILL_ALL)
    images = batch.render([gpu.View(0, w, h, 1, 9, cam), gpu.View(1, w, h, 1, 9, cam), gpu.View(1, w, h, 1, 9, cam)])[0]
    acc = np.zeros((h, w, 3), np.float32)
    osc.render(cam.as_array(), w, h, 9, rng_order=orc.RNG_GROUP, traversal=1, accum=acc)
    for image in images[1:]:
        assert (np.asarray(image) == orc.resolve(acc, 1)).all()
