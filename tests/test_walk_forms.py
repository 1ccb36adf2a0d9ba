"""A caller's BLAS as the walks see it (sofren2_gb300/csrc/sftg_walk.h, shared by the upload and the
kernels), on the CPU: child indices outside the tree, and the trees that may be expanded ahead of the
sequential walk."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sofren2_gb300", "csrc")

NODE = np.dtype([("mn", "<f4", (3, 8)), ("mx", "<f4", (3, 8)), ("child", "<u4", (8,)), ("count", "u1"), ("leaf", "u1"), ("pad", "u1", (30,))])
NONE, TRI = 0xFFFFFFFF, 0x80000000


@pytest.fixture(scope="module")
def walk_tool(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("walk") / "walk_forms")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC, os.path.join(ROOT, "tests", "walk_forms.cc"), "-o", exe], check=True)
    return exe


def run(exe, tmp_path, nodes, meshlets=2):
    path = str(tmp_path / "nodes.bin")
    nodes.tofile(path)
    return subprocess.run([exe, path, str(meshlets)], check=True, capture_output=True, text=True).stdout.splitlines()


def tree():
    """A root, two inner nodes and two leaves; every box inside its parent's."""
    n = np.zeros(5, NODE)
    n["mn"], n["mx"], n["child"] = 1e30, -1e30, NONE
    for i, kids, half in ((0, (1, 2), 4.0), (1, (3,), 2.0), (2, (4,), 2.0), (3, (TRI | 0, TRI | 129), 1.0), (4, (TRI | 127,), 1.0)):
        for c, ch in enumerate(kids):
            n[i]["mn"][:, c], n[i]["mx"][:, c], n[i]["child"][c] = -half, half, ch
        n[i]["count"], n[i]["leaf"] = len(kids), i >= 3
    return n


@pytest.mark.parametrize("bad", [5, 6, 1 << 20, (1 << 29) + 1, TRI - 1, TRI, TRI | 1, TRI | 4, TRI | 127, NONE - 1])
@pytest.mark.parametrize("node,slot", [(0, 0), (0, 1), (1, 0), (2, 7)])
def test_child_outside_the_tree_is_no_node_and_no_triangle(walk_tool, tmp_path, bad, node, slot):
    n = tree()
    n[node]["child"][slot] = bad
    words = [[int(w) for w in line.split()] for line in run(walk_tool, tmp_path, n)[:-1]]
    for i in range(len(n)):
        for c in range(8):
            if (i, c) == (node, slot):
                assert len(n) <= words[i][c] < TRI
            else:
                assert words[i][c] == n[i]["child"][c]


def test_sound_tree_keeps_its_words(walk_tool, tmp_path):
    n = tree()
    words = [[int(w) for w in line.split()] for line in run(walk_tool, tmp_path, n)[:-1]]
    assert np.array_equal(np.array(words, np.uint32), n["child"])


def nested(*args):
    return int(run(*args)[-1])


def test_sound_tree_is_nested(walk_tool, tmp_path):
    n = tree()
    n[4]["child"][5] = TRI | 300     # past the node's count: no slot of it
    n[1]["child"][2] = 77
    assert nested(walk_tool, tmp_path, n) == 1
    n[1]["count"], n[1]["child"][2] = 3, NONE     # counted, but empty
    assert nested(walk_tool, tmp_path, n) == 1


@pytest.mark.parametrize("node,slot,bad", [(0, 1, 5), (0, 0, TRI), (1, 0, TRI | 4), (2, 0, NONE - 1), (3, 1, TRI | 256), (4, 0, TRI | 1 << 20),
                                           (4, 0, NONE - 1)])
def test_tree_with_an_index_outside_the_model_is_not_nested(walk_tool, tmp_path, node, slot, bad):
    n = tree()
    n[node]["child"][slot] = bad
    assert nested(walk_tool, tmp_path, n) == 0


@pytest.mark.parametrize("field,value", [("mn", -4.5), ("mx", 4.5), ("mn", np.nan), ("mx", np.inf)])
@pytest.mark.parametrize("node", [1, 4])
def test_box_outside_its_parents_is_not_nested(walk_tool, tmp_path, node, field, value):
    n = tree()
    n[node][field][1, 0] = value
    assert nested(walk_tool, tmp_path, n) == 0
