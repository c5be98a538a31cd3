"""What scene creation reads of a caller's tree (scene_tree.h), compiled for the
host with the address and undefined-behaviour sanitizers: nodes that the roots
do not reach may hold anything.
"""

import os
import shutil
import subprocess

import numpy as np
import pytest

from convector_gb300 import scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "scene_tree.h"
int main(int, char** v) {
    std::FILE* f = std::fopen(v[1], "rb");
    unsigned n = 0, tris = 0;
    if (!f || std::fread(&n, 4, 1, f) != 1 || std::fread(&tris, 4, 1, f) != 1) return 2;
    std::vector<cvx_bvh_node> nodes(n);
    if (std::fread(nodes.data(), sizeof(cvx_bvh_node), n, f) != n) return 2;
    std::fclose(f);
    cvx::TreeFacts t;
    const char* wrong = cvx::check_tree(nodes.data(), n, tris, &t);
    if (wrong) return std::printf("refused: %s\n", wrong), 0;
    unsigned reached = 0;
    for (unsigned p = 0; p < n / 2; p++) reached += t.reached(p) ? 1u : 0u;
    std::printf("depth %u select %d wide %d reached %u\n", t.depth, (int)t.select, (int)t.wide, reached);
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    if shutil.which(cxx) is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("tree")
    (d / "main.cpp").write_text(PROGRAM)
    exe = str(d / "check")
    base = [cxx, "-std=c++17", "-g", "-O1", "-I", os.path.join(ROOT, "convector_gb300", "csrc"), "-o", exe,
            str(d / "main.cpp")]
    checked = ["-fsanitize=address,undefined", "-fno-sanitize-recover=all"]
    if subprocess.run(base + checked, capture_output=True).returncode != 0:  # no sanitizer runtime
        subprocess.run(base, check=True)

    def run(nodes, n_tris):
        (d / "tree").write_bytes(np.array([nodes.shape[0], n_tris], np.uint32).tobytes() + nodes.tobytes())
        r = subprocess.run([exe, str(d / "tree")], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout.strip()

    return run


@pytest.fixture(scope="module")
def built(cvx):
    b = cvx.Bvh.build(scenes.spheres_and_boxes(600, 5, obj=False)[0])
    return b.nodes, b.triangles.shape[0], b.depth


def test_built_tree(check, built):
    nodes, n, depth = built
    assert check(nodes, n) == "depth %d select 1 wide 1 reached %d" % (depth, nodes.shape[0] // 2)


@pytest.mark.parametrize("index,length", [(0xFFFFFFFE, 0), (0x7FFFFFFE, 0), (5, 0), (0, 0), (0xFFFFFFFF, 40)])
@pytest.mark.parametrize("bound", [0.0, np.nan, 3.0e38])
def test_unreached_nodes_are_not_followed(check, built, index, length, bound):
    """Padding behind the tree changes nothing about it."""
    nodes, n, depth = built
    pad = np.zeros((4, 8), np.uint32)
    pad.view(np.float32)[:, :6] = bound
    pad[:, 6:8] = (index, length)
    assert check(np.concatenate([nodes, pad]), n) == "depth %d select 1 wide 1 reached %d" % (depth, nodes.shape[0] // 2)


def test_forms(check, built):
    nodes, n, depth = built
    for at, value, want in ((0, -5.0, "select 1 wide 0"),            # a root wider than its children
                            (0, -1.0e30, "select 1 wide 0"),         # beyond the wide records' bound
                            (0, 1.0e30, "select 0 wide 0"),          # lo above hi
                            (3, np.inf, "select 0 wide 0")):
        v = nodes.copy()
        v.view(np.float32)[0, at] = value
        assert want in check(v, n)
    v = nodes.copy()
    v[0, 6:8] = (nodes.shape[0], 0)
    assert check(v, n).startswith("refused")
    v[0, 6:8] = (0xFFFFFFFE, 0)
    assert check(v, n).startswith("refused")
