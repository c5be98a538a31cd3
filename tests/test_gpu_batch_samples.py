"""Batches whose octet waves hold several samples of a view: every image equals
the same view rendered alone, sample by sample, on both sides of a wave's 16
samples, with views of unlike sample counts, in the kernel organisations a
batch mixes, and with captured graphs.
"""

import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("traversal", [0, 1])
@pytest.mark.parametrize("refill,mixed,graph", [(2, False, 0), (0, False, 1), (0, True, 0), (1, False, 0)])
def test_batch_samples_equal_alone(gpu, traversal, refill, mixed, graph):
    scs = [gpu.Scene(gpu.Bvh.build(scenes.spheres_and_boxes(n, 7, obj=False)[0])) for n in (500, 1500)]
    views = []
    for i, (w, h, spp) in enumerate([(64, 48, 16), (33, 17, 17), (1, 1, 1), (80, 20, 33), (16, 4, 2)]):
        cam = scenes.default_camera(gpu.Camera(), eye=(0.2 * i - 0.4, 1.2, 1.6))
        views.append(gpu.View(i % 2, w, h, spp, 0xFFFFFFF8 + i, cam))  # the frame numbers wrap
    batch = gpu.Batch(scs, max_groups=1 << 12, max_pixels=1 << 14, traversal=traversal, mode=gpu.MODE_MEGAKERNEL,
                      refill_mode=refill, use_graph=graph)
    if mixed:
        gpu.lib().cvx_batch_set_scene_mode(batch._h, 1, 1)
    for _ in range(2):
        imgs, rays, _ = batch.render(views)
        total = 0
        for v, img in zip(views, imgs):
            r = gpu.Renderer(scs[v.scene], v.width, v.height, rng_order=gpu.RNG_GROUP, traversal=traversal)
            r.set_camera(v.camera)
            for s in range(v.spp):
                r.accumulate_frame_f32((v.frame_base + s) & 0xFFFFFFFF)
                total += r.stats()[0]
            assert (img == r.resolve_u8(v.spp)).all()
        assert rays == total


def test_fused_views_behind_a_large_clear(gpu):
    """Fused views whose pixels lie behind many of wavefront views (cleared last), rendered twice into one
    batch's accumulator: each image equals the view's alone."""
    scs = [gpu.Scene(gpu.Bvh.build(scenes.spheres_and_boxes(n, 7, obj=False)[0])) for n in (500, 1500)]
    cam = scenes.default_camera(gpu.Camera(), eye=(0.1, 1.2, 1.6))
    views = [gpu.View(0, 4096, 4096, 1, 3, cam)] + [gpu.View(1, 64, 48, 2, 5 + i, cam) for i in range(3)]
    batch = gpu.Batch(scs, max_groups=1 << 22, max_pixels=(1 << 24) + 3 * 64 * 48, mode=gpu.MODE_MEGAKERNEL)
    gpu.lib().cvx_batch_set_scene_mode(batch._h, 0, 1)
    for _ in range(2):
        imgs = batch.render(views)[0]
        for v, img in zip(views[1:], imgs[1:]):
            r = gpu.Renderer(scs[1], v.width, v.height, rng_order=gpu.RNG_GROUP, traversal=gpu.TRAVERSE_SINGLE)
            r.set_camera(v.camera)
            r.accumulate_frames_f32(v.frame_base, v.spp)
            assert (img == r.resolve_u8(v.spp)).all()
