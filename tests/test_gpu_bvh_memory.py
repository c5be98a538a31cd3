"""A device-built BVH holds the memory of its arrays, not of the most nodes it might have had."""

import ctypes

import pytest

from convector_gb300 import scenes

pytestmark = pytest.mark.gpu


def _resident():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) * 1024 for line in f if line.startswith("VmRSS"))


def test_device_build_keeps_no_spare_nodes(gpu):
    tris = scenes.random_walk_tube(rings=600, obj=False)[0]
    n, lib = tris.shape[0], gpu.lib()

    def build():
        h = ctypes.c_void_p()
        gpu._check(lib.cvx_bvh_build_device(gpu._ptr(tris), n, ctypes.byref(h)))
        return h

    held = [build(), build()]  # the allocator and the driver have what they need
    nodes = lib.cvx_bvh_num_nodes(held[0])
    assert 32 * nodes < 0.7 * 64 * n  # else this would show nothing
    before = _resident()
    held += [build() for _ in range(6)]
    each = (_resident() - before) / 6
    exact = 32 * nodes + (64 + 4) * n
    for h in held:
        lib.cvx_bvh_destroy(h)
    # Half of what the spare nodes would take, for what else the process does.
    assert each < exact + 0.5 * (64 * n - 32 * nodes), (each, exact, n, nodes)
