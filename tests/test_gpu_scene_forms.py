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
