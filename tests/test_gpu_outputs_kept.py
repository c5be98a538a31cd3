"""A caller's image that a failed call does not fill stays as it was, to the last
byte (images of several pages each).
"""

import ctypes

import numpy as np
import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu

W, H, CVX_ERR_DEVICE = 400, 330, 6


@pytest.fixture(scope="module")
def scene(gpu):
    return gpu.Scene(gpu.Bvh.build(scenes.spheres_and_boxes(3000, 5, obj=False)[0]))


@pytest.fixture
def low_stack(gpu):
    gpu.set_traversal_stack_limit(2)
    yield
    gpu.set_traversal_stack_limit(0)


def _pattern(seed):
    return np.random.default_rng(seed).integers(0, 1 << 32, (H, W), dtype=np.uint32)


@pytest.mark.parametrize("kernel_mode,samples_per_wave", [(1, 1), (1, 4), (2, 1)])
def test_server_image_of_a_failed_request(gpu, scene, low_stack, kernel_mode, samples_per_wave):
    cam = scenes.default_camera(gpu.Camera())
    server = gpu.Server([scene], framebuffer_bytes=64 << 20, max_groups=1 << 16, kernel_mode=kernel_mode,
                        refill_mode=gpu.REFILL_ALL, samples_per_wave=samples_per_wave)
    img, rid, res = _pattern(1), ctypes.c_uint64(), gpu._Result()
    req = gpu._Request(0, W, H, 1, 3, cam._c)
    gpu._check(gpu.lib().cvx_server_submit(server._h, ctypes.byref(req), gpu._ptr(img), ctypes.byref(rid)))
    gpu._check(gpu.lib().cvx_server_wait(server._h, rid.value, 60000, ctypes.byref(res)))
    server.close()
    assert res.status == CVX_ERR_DEVICE
    assert (img == _pattern(1)).all()


@pytest.mark.parametrize("mode", [0, 1])
def test_batch_images_of_a_failed_call(gpu, scene, low_stack, mode):
    cam = scenes.default_camera(gpu.Camera())
    batch = gpu.Batch([scene], max_groups=1 << 16, max_pixels=2 * W * H, mode=mode)
    views = (gpu._View * 2)(*[gpu.View(0, W, H, 1 + i, 3, cam)._c() for i in range(2)])
    imgs = [_pattern(i) for i in range(2)]
    ptrs = (ctypes.c_void_p * 2)(*[im.ctypes.data for im in imgs])
    st = gpu.lib().cvx_batch_render(batch._h, views, 2, ptrs, None, None)
    assert st == CVX_ERR_DEVICE
    for i, img in enumerate(imgs):
        assert (img == _pattern(i)).all()
