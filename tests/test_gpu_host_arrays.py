"""Host arrays that a kernel cannot take in place, or not in any order: unaligned
ones and outputs that lie over inputs or over one another. Each call must give
what it gives for separate aligned arrays.
"""

import numpy as np
import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu


def _unaligned(a, by=1):
    """A copy of `a` whose data starts `by` bytes behind a multiple of 16."""
    raw = np.zeros(a.nbytes + 32, np.uint8)
    at = (-raw.ctypes.data) % 16 + by
    out = raw[at:at + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


def _same(a, b):
    return (a.view(np.uint32) == b.view(np.uint32)).all()


@pytest.fixture(scope="module")
def scene(gpu):
    return gpu.Scene(gpu.Bvh.build(scenes.spheres_and_boxes(600, 5, obj=False)[0]))


@pytest.mark.parametrize("traversal", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 3001, 131073])
@pytest.mark.parametrize("which", ["rays", "t", "tri", "all"])
def test_unaligned_query_arrays(gpu, scene, n, traversal, which):
    o, d = scenes.random_rays(n, seed=n)
    t, tri = scene.intersect_nearest(o, d, traversal=traversal)
    cols = [np.ascontiguousarray(a[:, k]) for a in (o, d) for k in range(3)]
    out_t, out_tri = np.zeros(n, np.float32), np.zeros(n, np.int32)
    if which in ("rays", "all"):
        cols = [_unaligned(c, 1 + k % 3) for k, c in enumerate(cols)]
    if which in ("t", "all"):
        out_t = _unaligned(out_t, 2)
    if which in ("tri", "all"):
        out_tri = _unaligned(out_tri, 3)
    gpu._check(gpu.lib().cvx_intersect_nearest(scene._h, *[gpu._ptr(c) for c in cols], n, 1.0e5, traversal,
                                               gpu._ptr(out_t), gpu._ptr(out_tri)))
    assert (np.array(out_tri) == tri).all() and _same(np.array(out_t), t)


@pytest.mark.parametrize("traversal", [0, 1])
@pytest.mark.parametrize("shift", [0, 1, -7])
def test_query_outputs_over_one_another(gpu, scene, traversal, shift):
    """One buffer for distances and indices, exactly or shifted: the indices are written last."""
    n = 3001
    o, d = scenes.random_rays(n, seed=4)
    t, tri = scene.intersect_nearest(o, d, traversal=traversal)
    cols = [np.ascontiguousarray(a[:, k]) for a in (o, d) for k in range(3)]
    buf = np.zeros(n + 7, np.uint32)
    at = max(-shift, 0)
    want = buf.copy()
    want[at:at + n] = t.view(np.uint32)
    want[at + shift:at + shift + n] = tri.view(np.uint32)
    gpu._check(gpu.lib().cvx_intersect_nearest(scene._h, *[gpu._ptr(c) for c in cols], n, 1.0e5, traversal,
                                               gpu._ptr(buf[at:]), gpu._ptr(buf[at + shift:])))
    assert (buf == want).all()


@pytest.mark.parametrize("w,h", [(1, 1), (33, 9), (31, 7), (64, 16), (65, 17)])
@pytest.mark.parametrize("form", ["aligned", "inputs unaligned", "output unaligned", "output over the frame",
                                  "output over the gbuffer"])
def test_display_arrays(gpu, orc, w, h, form):
    """Sizes around the filter's 32 x 8 tiles, with each array in place or copied."""
    rng = np.random.default_rng(w)
    tex = [rng.integers(0, 256, (8, 8, 3), dtype=np.uint8) for _ in range(2)]
    disp, od = gpu.Display(w, h, *tex), orc.OracleDisplay(w, h, *tex)
    for frame in range(9):  # more than the ring's eight
        rgba = rng.integers(0, 1 << 24, (h, w), dtype=np.uint32)
        gb = rng.integers(0, 1 << 24, (h, w), dtype=np.uint32) | (rng.integers(0, 3, (h, w), dtype=np.uint32) << 24)
        median = frame % 3 != 1
        ref = od.frame(rgba, gb, blend=True, median=median)
        a, g, out = rgba, gb, np.zeros((h, w), np.uint32)
        if form == "inputs unaligned":
            a, g = _unaligned(rgba, 1), _unaligned(gb, 2)
        if form == "output unaligned":
            out = _unaligned(out, 3)
        if form == "output over the frame":
            out = a = rgba.copy()
        if form == "output over the gbuffer":
            out = g = gb.copy()
        gpu._check(gpu.lib().cvx_display_frame(disp._h, gpu._ptr(a), gpu._ptr(g), 1, int(median), gpu._ptr(out)))
        assert (np.array(out) == ref).all(), (frame, np.count_nonzero(np.array(out) != ref))


def test_display_wrapper_takes_unaligned_arrays(gpu):
    w, h = 40, 12
    rng = np.random.default_rng(2)
    tex = [rng.integers(0, 256, (8, 8, 3), dtype=np.uint8) for _ in range(2)]
    rgba, gb = (rng.integers(0, 1 << 24, (h, w), dtype=np.uint32) for _ in range(2))
    raw = b"x" + rgba.tobytes() + gb.tobytes()
    a = np.frombuffer(raw, np.uint32, h * w, offset=1).reshape(h, w)
    g = np.frombuffer(raw, np.uint32, h * w, offset=1 + 4 * h * w).reshape(h, w)
    assert (gpu.Display(w, h, *tex).display_buffer(a, g) == gpu.Display(w, h, *tex).display_buffer(rgba, gb)).all()
